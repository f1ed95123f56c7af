// BEM assembly kernels for sm_103a: HeadMat blocks (S, D, N, deflation),
// DipSourceMat, the sensor matrices and the triangle preprocessing they share.
//
// Layout in HBM.  The head matrix lives as a dense N x N column-major FP64
// array in the solver's internal numbering -- triangle unknowns first, then
// vertex unknowns (the reference's [V | P] order rotated by n_vertices) --
// and only its lower triangle is written.  Per-triangle records (OperatorS
// data, P1 single-layer data, quadrature points) are precomputed once; the
// mixed far field stages them tile by tile into shared memory with bulk (TMA)
// copies, the FP64 S and D blocks read tables of distances and edge integrals.
//
// The integrals are the reference's: its analytic inner integral under its
// Gauss outer rule, so the FP64 results agree with it to rounding.
#include <algorithm>
#include <cstdio>
#include <string>
#include <tuple>
#include <vector>

#include "device_common.cuh"
#include "fixed64.cuh"
#include "handles.h"
#include "omg_internal.h"

namespace omg {

using dev::d3;

// Gauss rules of 3/6/7/16 points (OpenMEEG/include/integrator.h:260-318;
// Bonnet's tables).  The digits are those of the reference: parity at 1e-10
// requires the same truncated nodes.  [order][point] = {b0, b1, b2, weight}.
__constant__ double c_rules[4][16][4] = {
    {{0.166666666666667, 0.166666666666667, 0.666666666666667, 0.333333333333334},
     {0.166666666666667, 0.666666666666667, 0.166666666666667, 0.333333333333334},
     {0.666666666666667, 0.166666666666667, 0.166666666666667, 0.333333333333334}},
    {{0.445948490915965, 0.445948490915965, 0.108103018168070, 0.223381589678010},
     {0.445948490915965, 0.108103018168070, 0.445948490915965, 0.223381589678010},
     {0.108103018168070, 0.445948490915965, 0.445948490915965, 0.223381589678010},
     {0.091576213509771, 0.091576213509771, 0.816847572980458, 0.109951743655322},
     {0.091576213509771, 0.816847572980458, 0.091576213509771, 0.109951743655322},
     {0.816847572980458, 0.091576213509771, 0.091576213509771, 0.109951743655322}},
    {{0.333333333333333, 0.333333333333333, 0.333333333333333, 0.2250},
     {0.470142064105115, 0.470142064105115, 0.059715871789770, 0.132394152788506},
     {0.470142064105115, 0.059715871789770, 0.470142064105115, 0.132394152788506},
     {0.059715871789770, 0.470142064105115, 0.470142064105115, 0.132394152788506},
     {0.101286507323456, 0.101286507323456, 0.797426985353088, 0.125939180544828},
     {0.101286507323456, 0.797426985353088, 0.101286507323456, 0.125939180544828},
     {0.797426985353088, 0.101286507323456, 0.101286507323456, 0.125939180544828}},
    {{0.333333333333333, 0.333333333333333, 0.333333333333333, 0.144315607677786},
     {0.081414823414554, 0.459292588292722, 0.459292588292722, 0.095091634267284},
     {0.459292588292722, 0.081414823414554, 0.459292588292722, 0.095091634267284},
     {0.459292588292722, 0.459292588292722, 0.081414823414554, 0.095091634267284},
     {0.898905543365937, 0.050547228317031, 0.050547228317031, 0.032458497623198},
     {0.050547228317031, 0.898905543365937, 0.050547228317031, 0.032458497623198},
     {0.050547228317031, 0.050547228317031, 0.898905543365937, 0.032458497623198},
     {0.658861384496479, 0.170569307751760, 0.170569307751761, 0.103217370534718},
     {0.170569307751760, 0.658861384496479, 0.170569307751761, 0.103217370534718},
     {0.170569307751760, 0.170569307751761, 0.658861384496479, 0.103217370534718},
     {0.008394777409957, 0.728492392955404, 0.263112829634639, 0.027230314174434},
     {0.728492392955404, 0.008394777409957, 0.263112829634639, 0.027230314174434},
     {0.728492392955404, 0.263112829634639, 0.008394777409957, 0.027230314174434},
     {0.008394777409957, 0.263112829634639, 0.728492392955404, 0.027230314174434},
     {0.263112829634639, 0.008394777409957, 0.728492392955404, 0.027230314174434},
     {0.263112829634639, 0.728492392955404, 0.008394777409957, 0.027230314174434}}};
__constant__ int c_nbpts[4] = {3, 6, 7, 16};

static int64_t g_launches = 0;
int64_t kernel_launch_count() { return g_launches; }
void count_launch(int n) { g_launches += n; }

// ---- launch profiler (events pooled; aggregated on read) ----
struct ProfEntry {
    const char* name;
    cudaEvent_t a, b;
};
static bool g_prof = false;
static std::vector<ProfEntry> g_prof_entries;
static std::vector<cudaEvent_t> g_prof_pool;
bool profiling_enabled() { return g_prof; }
cudaEvent_t profile_event() {
    if (!g_prof_pool.empty()) {
        cudaEvent_t e = g_prof_pool.back();
        g_prof_pool.pop_back();
        return e;
    }
    cudaEvent_t e;
    cudaEventCreate(&e);
    return e;
}
void profile_record(const char* name, cudaEvent_t a, cudaEvent_t b) { g_prof_entries.push_back({name, a, b}); }
void profile_enable(bool on) { g_prof = on; }
// Aggregates recorded launches per name (synchronizes on each event).
std::vector<std::tuple<std::string, int64_t, double>> profile_collect() {
    std::vector<std::tuple<std::string, int64_t, double>> out;
    for (auto& e : g_prof_entries) {
        cudaEventSynchronize(e.b);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e.a, e.b);
        bool found = false;
        for (auto& o : out)
            if (std::get<0>(o) == e.name) {
                std::get<1>(o) += 1;
                std::get<2>(o) += ms;
                found = true;
            }
        if (!found) out.emplace_back(e.name, 1, (double)ms);
        g_prof_pool.push_back(e.a);
        g_prof_pool.push_back(e.b);
    }
    g_prof_entries.clear();
    return out;
}

static inline void check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw Error(OMG_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
    count_launch();
}

static inline unsigned nblocks(int64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

// Quadrature point: sum_j b_j p_j accumulated from zero without contraction,
// as Vect3::multadd does (integrator.h:214-225).
__device__ __forceinline__ d3 bary_point(const double* r, d3 p0, d3 p1, d3 p2) {
    d3 v;
    v.x = __dadd_rn(__dadd_rn(__dmul_rn(r[0], p0.x), __dmul_rn(r[1], p1.x)), __dmul_rn(r[2], p2.x));
    v.y = __dadd_rn(__dadd_rn(__dmul_rn(r[0], p0.y), __dmul_rn(r[1], p1.y)), __dmul_rn(r[2], p2.y));
    v.z = __dadd_rn(__dadd_rn(__dmul_rn(r[0], p0.z), __dmul_rn(r[1], p1.z)), __dmul_rn(r[2], p2.z));
    return v;
}

// ---------------------------------------------------------------------------
// Triangle preprocessing: normal/area (triangle.h:57-62), OperatorS edge data
// (analytics.h:22-30), P1SingleLayerPotential edge data (analytics.h:81-85),
// and the points of the `order` rule.
// ---------------------------------------------------------------------------
__global__ void prepare_triangles_kernel(int64_t nt, const double* __restrict__ V, const int32_t* __restrict__ T,
                                         int order, double* srec, double* prec, double* qrec) {
    int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const d3 p0 = dev::ld3(V + 3 * (int64_t)T[3 * t]);
    const d3 p1 = dev::ld3(V + 3 * (int64_t)T[3 * t + 1]);
    const d3 p2 = dev::ld3(V + 3 * (int64_t)T[3 * t + 2]);
    d3 nn = dev::cross(p1 - p0, p2 - p0);
    const double nrm = dev::norm(nn);
    const double area = 0.5 * nrm;
    const d3 n = nn * (1.0 / nrm);
    double* s = srec + t * SREC;
    const d3 P[3] = {p0, p1, p2};
    for (int i = 0; i < 3; ++i) {
        s[3 * i] = P[i].x;
        s[3 * i + 1] = P[i].y;
        s[3 * i + 2] = P[i].z;
    }
    s[9] = n.x; s[10] = n.y; s[11] = n.z;
    s[12] = area;
    for (int i = 0; i < 3; ++i) {
        const d3 vref = P[i] - P[(i + 1) % 3];
        const double len = dev::norm(vref);
        const d3 unit = dev::mk(vref.x / len, vref.y / len, vref.z / len);
        const d3 en = dev::cross(n, unit);
        s[13 + i] = len;
        s[16 + 3 * i] = en.x; s[17 + 3 * i] = en.y; s[18 + 3 * i] = en.z;
    }
    for (int i = 25; i < SREC; ++i) s[i] = 0.0;
    double* p = prec + t * PREC;
    for (int i = 0; i < 13; ++i) p[i] = s[i];
    const d3 D[3] = {p1 - p0, p2 - p1, p0 - p2};
    for (int i = 0; i < 3; ++i) {
        const double dn = dev::norm(D[i]);
        p[13 + 3 * i] = D[i].x; p[14 + 3 * i] = D[i].y; p[15 + 3 * i] = D[i].z;
        p[22 + 3 * i] = D[i].x / dn; p[23 + 3 * i] = D[i].y / dn; p[24 + 3 * i] = D[i].z / dn;
    }
    p[31] = 0.0;
    double* q = qrec + t * QREC;
    const int np = c_nbpts[order];
    for (int k = 0; k < MAXQ; ++k) {
        d3 v = dev::mk(0, 0, 0);
        if (k < np) v = bary_point(c_rules[order][k], p0, p1, p2);
        q[3 * k] = v.x; q[3 * k + 1] = v.y; q[3 * k + 2] = v.z;
    }
    q[48] = area;
    for (int i = 49; i < QREC; ++i) q[i] = 0.0;
}

void launch_prepare_triangles_order(const DevGeom& g, int order, cudaStream_t s) {
    ProfScope prof_("prepare_triangles", s);
    prepare_triangles_kernel<<<nblocks(g.nt, 128), 128, 0, s>>>(g.nt, g.V, g.T, order, g.srec, g.prec, g.qrec);
    check_launch("prepare_triangles");
}
void launch_prepare_triangles(const DevGeom& g, cudaStream_t s) { launch_prepare_triangles_order(g, 3, s); }

// Lower-triangle address of (a, b) in the internal column-major matrix.
__device__ __forceinline__ int64_t lower_at(int64_t a, int64_t b, int64_t ld) {
    return a >= b ? a + b * ld : b + a * ld;
}

// ---------------------------------------------------------------------------
// S and D blocks (DiagonalBlock::S operators.h:209-237, NonDiagonalBlock::S
// :391-425, BlocksBase::D :83-115) in FP64:
//   S(b, a) = integral over a (Gauss rule) of OperatorS(b),
//   D(a, b, j) = integral over a of P1SingleLayerPotential(b)_j,
// for the analytic triangles b of one mesh and the rule points of the
// triangles a of another (or the same) one.
//
// The FP64 pipe bounds these blocks (one thread per pair evaluating both closed
// forms from their vertices kept it 88% busy: ~270 operations per single-layer
// value, ~300 per double-layer one), so the operations are shared as far as the
// closed forms allow, and memory traffic, which FP64 leaves nearly idle, is spent
// for it.  For a batch of points, three launches fill and read global tables:
//   1. d[v][x] = |x - v| for every vertex of the analytic mesh (half a vertex per
//      triangle, instead of three distances per triangle);
//   2. l[e][x] = (integral over the edge of 1/|x - y|) / length
//      = 2 atanh(len / (d_a + d_b)) / len for every edge (1.5 per triangle instead
//      of three logarithms each in S and in D: D's log((d_b + r_b.u)/(d_a + r_a.u))
//      is the same integral), and (d_a +- d_b)^2 - len^2 = 2 (r_a.r_b +- d_a d_b);
//   3. per (triangle, point): h = n.(p0 - x) and E_j = n.(r_j+1 x r_j+2) (linear in
//      x; E_0 + E_1 + E_2 = 2A), half the solid angle
//      w = atan(2 A h / (d0 d1 d2 + sum d_i r_j.r_k)), then
//        S = sum_i E_opp(i) l_i - 2 h w,
//        D_j = (w E_j + h/2 D_j+1.(sum_i D_i l_i)) / A, D_0 + D_1 + D_2 = 2 w,
//      in 16 operations with l_0 - l_1 and l_2 - l_1 (the D_i sum to zero).
// About 25 FP64 operations per (triangle, point) for S and D together.  The square
// roots, logarithms, arctangents, the weights of the rule and the linear forms h, E_j
// run on the integer pipe (fixed64.cuh), which issues beside the FP64 operations: the
// forms as inner products of 60-bit vectors, of the triangle and of x - p0 from the
// table.  A head matrix of four layers (7020 triangles) took 67 ms in these kernels
// with all of it in FP64 (75 operations), 34 with the linear forms in FP64 (35), now
// 22.5: the pair kernel holds the FP64 pipe 84% busy, the distances likewise, and the
// edges (285 instructions each, 29% of the time) issue 66% of what the SM can.
// Lanes run over the triangles a at the same rule point, so every table read is
// coalesced, the triangle b is uniform in a warp, and the sum over the rule stays
// in registers (no shuffles, which cost FP64 additions).
// ---------------------------------------------------------------------------
// Record of an analytic triangle: -2 N, N x D0, N x D2 (N = D0 x (p2 - p0), |N| = 2A; in block fixed point, 3 each; their
// exponents in an int4 of their own table), 4A^2, |D0|^2 / 4, |D2|^2 / 4,
// D0.D2 / 4, the bits of 2e-10 * 2A, 1 / 2A, 2 / 4A^2, |D_i|^2 (3), |D_i| (3)
constexpr int TGEO = 22;

// v in block fixed point; returns its exponent.
__device__ __forceinline__ int sd_fix(d3 v, int2* out) {
    const int ex = (int)fx::expo(v.x), ey = (int)fx::expo(v.y), ez = (int)fx::expo(v.z), em = max(ex, max(ey, ez));
    out[0] = fx::limbs(fx::fix60(v.x, em - ex));
    out[1] = fx::limbs(fx::fix60(v.y, em - ey));
    out[2] = fx::limbs(fx::fix60(v.z, em - ez));
    return em - 1022;
}

__global__ void sd_geometry_kernel(int64_t t0, int64_t nt, const double* __restrict__ V,
                                   const int32_t* __restrict__ T, const int32_t* __restrict__ v2t_beg,
                                   const int32_t* __restrict__ v2t_tri, double* tgeo, int4* gexp, int32_t* eown) {
    const int64_t it = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (it >= nt) return;
    const int32_t* tv = T + 3 * (t0 + it);
    const d3 p0 = dev::ld3(V + 3 * (int64_t)tv[0]), p1 = dev::ld3(V + 3 * (int64_t)tv[1]),
             p2 = dev::ld3(V + 3 * (int64_t)tv[2]);
    const d3 D0 = p1 - p0, D1 = p2 - p1, D2 = p0 - p2;
    const d3 nn = dev::cross(D0, p2 - p0);
    const d3 m0 = dev::cross(nn, D0), m2 = dev::cross(nn, D2);
    const double a22 = dev::dot(nn, nn), a2 = sqrt(a22);
    double* g = tgeo + it * TGEO;
    int2* gf = reinterpret_cast<int2*>(g);
    gexp[it] = make_int4(sd_fix(nn * -2.0, gf), sd_fix(m0, gf + 3), sd_fix(m2, gf + 6), 0);
    g[9] = a22;
    g[16] = dev::dot(D0, D0); g[17] = dev::dot(D1, D1); g[18] = dev::dot(D2, D2);
    g[10] = 0.25 * g[16]; g[11] = 0.25 * g[18]; g[12] = 0.25 * dev::dot(D2, D0);
    g[13] = 2e-10 * a2;
    g[14] = 1.0 / a2; g[15] = 2.0 / a22;
    g[19] = sqrt(g[16]); g[20] = sqrt(g[17]); g[21] = sqrt(g[18]);
    // table row of edge i (corners i, i + 1): the slot 3 t + i of the first triangle of the range that has it
    for (int i = 0; i < 3; ++i) {
        const int32_t a = tv[i], b = tv[(i + 1) % 3];
        int32_t own = (int32_t)(3 * it + i);
        for (int k = v2t_beg[a]; k < v2t_beg[a + 1]; ++k) {
            const int64_t t = v2t_tri[k];
            if (t < t0 || t >= t0 + it) continue;   // (triangles around a vertex are listed in increasing order)
            const int32_t* u = T + 3 * t;
            int found = -1;
            for (int j = 0; j < 3; ++j)
                if ((u[j] == a && u[(j + 1) % 3] == b) || (u[j] == b && u[(j + 1) % 3] == a)) found = j;
            if (found >= 0) {
                own = (int32_t)(3 * (t - t0) + found);
                break;
            }
        }
        eown[3 * it + i] = own;
    }
}

// 1/x to about an ulp: the hardware approximation y times the geometric series 1 + e + e^2 of 1 / (1 - e), e = 1 - x y.
__device__ __forceinline__ double sd_rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(fma(e, e, e), y, y);
}
// |x| / 2 < 1e-10 on the integer pipe.
__device__ __forceinline__ bool sd_flat2(double x) {
    return (__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFll) < __double_as_longlong(2e-10);
}
constexpr int SD_V = 8;      // vertices per CTA of the distance table
constexpr int SD_E = 4;       // triangles per CTA of the edge table
constexpr int SD_THREADS = 256;

// The CTAs of the three launches run over the points (or the triangles a) along x and over the analytic mesh along y and z:
// a source surface has more triangles than gridDim.y alone can hold (65535 CTAs, 131070 triangles).  One index over both
// directions, divided in the kernel, took 1.4% off the four-layer head.
constexpr unsigned SD_GRID_Y = 65535;
__device__ __forceinline__ unsigned sd_cta_y() { return blockIdx.z * SD_GRID_Y + blockIdx.y; }
static dim3 sd_grid(unsigned gx, unsigned gy) { return dim3(gx, std::min(gy, SD_GRID_Y), (gy + SD_GRID_Y - 1) / SD_GRID_Y); }

// Point x = q na + ia of a batch of na triangles from a0: point q of triangle a0 + ia.  For vertex vb + v: the distance
// d[v * npt + x] and, in the rows 3 v .. 3 v + 2 of cv, the point minus the vertex in block fixed point with E = the exponent
// of the distance + 1.
__global__ void __launch_bounds__(SD_THREADS) sd_distance_kernel(const double* __restrict__ qrec, int64_t a0, int na,
                                                                 int npt, const double* __restrict__ V, int64_t vb,
                                                                 int nv, int2* __restrict__ cv,
                                                                 double* __restrict__ d) {
    const int x = blockIdx.x * SD_THREADS + threadIdx.x;
    if (x >= npt) return;
    const int q = x / na, ia = x - q * na;
    const double* src = qrec + (a0 + ia) * QREC + 3 * q;
    const double px = src[0], py = src[1], pz = src[2];
    const int v0 = sd_cta_y() * SD_V, v1 = min(nv, v0 + SD_V);
#pragma unroll 4
    for (int v = v0; v < v1; ++v) {
        const double* p = V + 3 * (vb + v);
        const double rx = px - p[0], ry = py - p[1], rz = pz - p[2];
        const int64_t o = (int64_t)v * npt + x;
        const double dist = fx::sqrt64(fma(rx, rx, fma(ry, ry, rz * rz)));
        const int e = (int)fx::expo(dist);
        d[o] = dist;
        int2* c = cv + o + 2 * (int64_t)v * npt;
        c[0] = fx::limbs(fx::fix60(rx, e - (int)fx::expo(rx)));
        c[npt] = fx::limbs(fx::fix60(ry, e - (int)fx::expo(ry)));
        c[2 * (int64_t)npt] = fx::limbs(fx::fix60(rz, e - (int)fx::expo(rz)));
    }
}

// Row 3 b + i, edge i (corners i, i + 1) of triangle b, of the rows that own their edge: l times the point's weight, and in
// prod (d_a + d_b)^2 - len^2 = 2 (d_a d_b + r_a.r_b) and (d_a - d_b)^2 - len^2 = 2 (r_a.r_b - d_a d_b).
__global__ void __launch_bounds__(SD_THREADS) sd_edge_kernel(int64_t tb, int nb, int na, int npt, int order,
                                                             const int32_t* __restrict__ T, int64_t vb,
                                                             const double* __restrict__ tgeo,
                                                             const int32_t* __restrict__ eown,
                                                             const double* __restrict__ d, double* __restrict__ l,
                                                             double2* __restrict__ prod) {
    const int x = blockIdx.x * SD_THREADS + threadIdx.x;
    if (x >= npt) return;
    const double wr = c_rules[order][x / na][3];
    const uint64_t wm = fx::mant(wr);
    const int we = (int)fx::expo(wr);
    const int b0 = sd_cta_y() * SD_E, b1 = min(nb, b0 + SD_E);
    for (int b = b0; b < b1; ++b) {
        const int32_t* tv = T + 3 * (tb + b);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (eown[3 * b + i] != 3 * b + i) continue;
            const double da = d[(int64_t)(tv[i] - vb) * npt + x], db = d[(int64_t)(tv[i == 2 ? 0 : i + 1] - vb) * npt + x];
            const double R = da + db;
            l[(int64_t)(3 * b + i) * npt + x] = fx::edge<true>(R, tgeo[b * (int64_t)TGEO + 19 + i], wm, we, wr);
            const double q = tgeo[b * (int64_t)TGEO + 16 + i], D = da - db;
            prod[(int64_t)(3 * b + i) * npt + x] = make_double2(fma(R, R, -q), fma(D, D, -q));
        }
    }
}

// The pairs (triangle b, triangle a0 + ia of the batch): warp w of a CTA holds b, its lanes 32 triangles a.
// S for a >= b only when `same`.
// CTAs of two warps: a small head fills more SMs evenly (the smallest gain's blocks 1.26 ms, 1.5 with four warps, 1.6 with
// eight); 8 CTAs of 105 registers (more, with fewer registers, were no faster).
constexpr int SD_WARPS = 2, SD_CTAS = 8;
template <bool WANT_S, bool WANT_D>
__global__ void __launch_bounds__(32 * SD_WARPS, SD_CTAS) sd_pair_kernel(
    int64_t tb, int nb, unsigned gy, unsigned first, int64_t ta, int64_t a0, int na, int npt, int order, int same, double coeff,
    const int32_t* __restrict__ T, int64_t vb, const double* __restrict__ tgeo, const int4* __restrict__ gexp,
    const int32_t* __restrict__ eown, const double* __restrict__ qrec, const int2* __restrict__ cv,
    const double* __restrict__ d,
    const double* __restrict__ l, const double2* __restrict__ prod, const int32_t* __restrict__ tpos, double* hm,
    int64_t ld, double* stmp, int64_t n2, double* dtmp) {
    if (sd_cta_y() >= gy) return;
    const unsigned by = sd_cta_y() + first;
    const int b = (by < gy ? by : by - gy) * SD_WARPS + threadIdx.x / 32;
    if (b >= nb) return;
    const int lane_a = blockIdx.x * 32 + threadIdx.x % 32;
    const bool live = lane_a < na;
    const int ia = live ? lane_a : na - 1;
    const int64_t a = a0 + ia;   // relative to ta
    const bool wantS = WANT_S && (!same || a >= b);
    if (!WANT_D && !__any_sync(0xffffffffu, wantS)) return;
    const double* g = tgeo + (int64_t)b * TGEO;
    const int2* gf = reinterpret_cast<const int2*>(g);
    const int2 nx = gf[0], ny = gf[1], nz = gf[2], m0x = gf[3], m0y = gf[4], m0z = gf[5], m2x = gf[6], m2y = gf[7],
               m2z = gf[8];
    const int4 ge = gexp[b];
    const double A4 = g[9];
    const long long flat = __double_as_longlong(g[13]);
    const int32_t* tv = T + 3 * (tb + b);
    const double* dr0 = d + (int64_t)(tv[0] - vb) * npt + ia;
    const double* dr1 = d + (int64_t)(tv[1] - vb) * npt + ia;
    const double* dr2 = d + (int64_t)(tv[2] - vb) * npt + ia;
    const int64_t x0 = (int64_t)eown[3 * b] * npt + ia, x1 = (int64_t)eown[3 * b + 1] * npt + ia,
                  x2 = (int64_t)eown[3 * b + 2] * npt + ia;
    const int2* cx = cv + 3 * (int64_t)(tv[0] - vb) * npt + ia;
    const int2* cy = cx + npt;
    const int2* cz = cy + npt;
    const int np = c_nbpts[order];
    const bool anyS = WANT_S && __any_sync(0xffffffffu, wantS);
    // times 2A: S; s_j of D without the terms h sum D_i l_i, whose sums over the rule are f0 (of l_0 - l_1) and f2 (l_2 - l_1)
    double sS = 0.0, s1 = 0.0, s2 = 0.0, sw = 0.0, f0 = 0.0, f2 = 0.0;
    for (int k = 0, o = 0; k < np; ++k, o += na) {
        const double d0 = dr0[o], d1 = dr1[o], d2 = dr2[o], l1 = l[x1 + o];
        const double m0 = l[x0 + o] - l1, m2 = l[x2 + o] - l1;
        const int2 x = cx[o], y = cy[o], z = cz[o];
        const int ce = (int)fx::expo(d0) - 1022;
        const double num = fx::value60(fx::dot60(nx, ny, nz, x, y, z), ge.x + ce);   // 2A 2h
        const double E2 = fx::value60(fx::dot60(m0x, m0y, m0z, x, y, z), ge.y + ce);
        const double E1 = fx::value60(fx::dot60(m2x, m2y, m2z, x, y, z), ge.z + ce);
        // 2 (d0 d1 d2 + sum d_i r_j.r_k) by the tabled 2 (r_j.r_k +- d_j d_k)
        const double den = fma(d0, prod[x1 + o].y, fma(d1, prod[x2 + o].x, d2 * prod[x0 + o].x));
        const double wr = c_rules[order][k][3];
        const double w = fx::half_angle<true>(num, den, fx::mant(wr), (int)fx::expo(wr), wr);
        if (anyS) {   // E0 = 2A - E1 - E2
            const double el = fma(A4, l1, fma(E2, m0, E1 * m2));   // (summed before sS: one rounding of the sum per point)
            sS += fma(-num, sd_flat2(num) ? 0.0 : w, el);
        }
        if (WANT_D && (__double_as_longlong(num) & 0x7FFFFFFFFFFFFFFFll) >= flat) {   // |2h| >= 2e-10
            s1 = fma(w, E1, s1);
            s2 = fma(w, E2, s2);
            sw += w;
            f0 = fma(num, m0, f0);
            f2 = fma(num, m2, f2);
        }
    }
    if (!live) return;
    const double area = qrec[(ta + a) * QREC + 48];
    if (wantS) {
        const double val = area * (g[14] * sS);
        if (hm) {
            hm[lower_at(tpos[tb + b], tpos[ta + a], ld)] = val * coeff;
        } else {
            stmp[b * n2 + a] = val;
            if (same) stmp[a * n2 + b] = val;
        }
    }
    if (WANT_D) {
        double* o = dtmp + (a * nb + b) * 3;
        const double iA = g[15];   // sum D_i l_i = D0 m0 + D2 m2; the components' sum is 2 w
        s1 = iA * fma(g[12], f0, fma(g[11], f2, s1));
        s2 = iA * fma(g[10], f0, fma(g[12], f2, s2));
        o[0] = area * (2.0 * sw - s1 - s2);
        o[1] = area * s1;
        o[2] = area * s2;
    }
}

// The blocks of the analytic triangles [tbb, tbe) (vertices [vbb, vbe)) and the rule points of the triangles
// [tab, tae).  wantS: S into hm (times coeff) or into the dense b-major stmp; `same`: one mesh against itself.
// dtmp: D, [a][b][3], or null.
void launch_SD_block(const DevGeom& g, int64_t tbb, int64_t tbe, int64_t vbb, int64_t vbe, int64_t tab, int64_t tae,
                     bool same, int order, bool wantS, double coeff, double* hm, int64_t ld, double* stmp,
                     double* dtmp, cudaStream_t s) {
    const int64_t nb = tbe - tbb, na = tae - tab, nv = vbe - vbb;
    if (nb <= 0 || na <= 0 || (!wantS && !dtmp)) return;
    ProfScope prof_("sd_block", s);
    if (nb > (1 << 28)) throw Error(OMG_ERR_UNSUPPORTED, "S / D block too large");
    constexpr int NPTS[4] = {3, 6, 7, 16};
    const int np = NPTS[order];
    // Points per batch: tables of about 2 GB, batches of equal size in multiples of 32 triangles (full warps).  A batch's
    // kernels each end with a part-empty last wave, which costs more than tables that stay in L2 would save: the four-layer
    // head takes 23.3 ms at 1 GB, 22.7 at 1.5, 22.5 here (with smaller tables 36.5 at 128 MB, 28.1 at 256, 25.4 at 512).
    const int64_t per_tri = (4 * nv + 9 * nb) * 8 * np;
    const int64_t most = std::max<int64_t>(32, std::min<int64_t>((2048ll << 20) / per_tri, 4096) / 32 * 32);
    const int64_t nbatch = (na + most - 1) / most, batch = std::min(na, ((na + nbatch - 1) / nbatch + 31) / 32 * 32);
    DevBuf geo((size_t)nb * (TGEO * 8 + 16 + 3 * 4), s), tab_((size_t)per_tri * batch, s);
    int4* gexp = geo.as<int4>();
    double* tgeo = reinterpret_cast<double*>(gexp + nb);
    int32_t* eown = reinterpret_cast<int32_t*>(tgeo + nb * TGEO);
    sd_geometry_kernel<<<nblocks(nb, 64), 64, 0, s>>>(tbb, nb, g.V, g.T, g.v2t_beg, g.v2t_tri, tgeo, gexp, eown);
    check_launch("S / D geometry");
    for (int64_t a0 = 0; a0 < na; a0 += batch) {
        const int n = (int)std::min(batch, na - a0), npt = n * np;
        double2* prod = tab_.as<double2>();
        int2* cv = reinterpret_cast<int2*>(prod + 3 * nb * npt);
        double* d = reinterpret_cast<double*>(cv + 3 * nv * npt);
        double* l = d + nv * npt;
        const unsigned gx = nblocks(npt, SD_THREADS);
        sd_distance_kernel<<<sd_grid(gx, nblocks(nv, SD_V)), SD_THREADS, 0, s>>>(g.qrec, tab + a0, n, npt, g.V, vbb, (int)nv,
                                                                               cv, d);
        check_launch("S / D distances");
        sd_edge_kernel<<<sd_grid(gx, nblocks(nb, SD_E)), SD_THREADS, 0, s>>>(tbb, (int)nb, n, npt, order, g.T, vbb, tgeo,
                                                                             eown, d, l, prod);
        check_launch("S / D edges");
        const unsigned py = nblocks(nb, SD_WARPS);
        // Triangles close to the batch's (the same part of the other mesh's numbering) take up to three times as long:
        // their CTAs are started first.
        const unsigned first = (unsigned)(a0 * py / na);
        auto kern = wantS ? (dtmp ? sd_pair_kernel<true, true> : sd_pair_kernel<true, false>) : sd_pair_kernel<false, true>;
        kern<<<sd_grid(nblocks(n, 32), py), 32 * SD_WARPS, 0, s>>>(tbb, (int)nb, py, first, tab, a0, n, npt, order, same ? 1 : 0, coeff,
                                                     g.T, vbb, tgeo, gexp, eown, g.qrec, cv, d, l, prod, g.tpos, hm, ld, stmp,
                                                     na, dtmp);
        check_launch("S / D pairs");
    }
}

// HM(t1, v) += coeff * sum over triangles t2 of B containing v of tmp[t1][t2][local(v)]
// (the += of operators.h:108-109, in increasing t2 order).
__global__ void d_gather_kernel(int64_t tab, int64_t na, int64_t tbb, int64_t nb, int64_t vbb, int64_t nvb,
                                double coeff, const double* __restrict__ tmp, const int32_t* __restrict__ v2t_beg,
                                const int32_t* __restrict__ v2t_tri, const int8_t* __restrict__ v2t_loc,
                                const int32_t* __restrict__ tpos, int64_t nP, double* hm, int64_t ld, int rect) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= na * nvb) return;
    const int64_t iv = idx % nvb, ia = idx / nvb;
    const int64_t v = vbb + iv;
    double sum = 0.0;
    for (int k = v2t_beg[v]; k < v2t_beg[v + 1]; ++k) {
        const int64_t t2 = v2t_tri[k];
        if (t2 < tbb || t2 >= tbb + nb) continue;
        sum += tmp[(ia * nb + (t2 - tbb)) * 3 + v2t_loc[k]];
    }
    if (rect)   // rectangular output: row = the triangle's unknown, column = the vertex within B
        hm[tpos[tab + ia] + iv * ld] += coeff * sum;
    else
        hm[lower_at(tpos[tab + ia], nP + v, ld)] += coeff * sum;
}

void launch_D_gather(const DevGeom& g, int64_t tab, int64_t tae, int64_t tbb, int64_t tbe, int64_t vbb, int64_t vbe,
                     double coeff, const double* tmp, double* hm, int64_t ld, cudaStream_t s, bool rect) {
    ProfScope prof_("d_gather", s);
    const int64_t n = (tae - tab) * (vbe - vbb);
    d_gather_kernel<<<nblocks(n, 256), 256, 0, s>>>(tab, tae - tab, tbb, tbe - tbb, vbb, vbe - vbb, coeff, tmp,
                                                    g.v2t_beg, g.v2t_tri, g.v2t_loc, g.tpos, g.nP, hm, ld,
                                                    rect ? 1 : 0);
    check_launch("D gather");
}

// ---------------------------------------------------------------------------
// N block (BlocksBase::N operators.h:119-148 through DiagonalBlock::N :271-296
// and NonDiagonalBlock::N :454-480):
//   N(v1,v2) = - sum_{t1 ∋ v1, t2 ∋ v2} f (CB1.CB2) S(t1,t2) / (A1 A2)
// with f = 1/4 (1/2 for the same vertex across meshes).  S comes from the head
// matrix (scaled by coeff/Scoeff) or from a temporary unit-coefficient block.
// ---------------------------------------------------------------------------
__device__ __forceinline__ d3 edge_cb(const double* V, const int32_t* T, int64_t t, int loc) {
    // Edge(V) opposite the vertex: vertices {1,2},{2,0},{0,1} (triangle.h:87-94,154)
    const int a = (loc + 1) % 3, b = (loc + 2) % 3;
    return dev::ld3(V + 3 * (int64_t)T[3 * t + a]) - dev::ld3(V + 3 * (int64_t)T[3 * t + b]);
}

// Per vertex-triangle slot (CSR of v2t): q = CB / A, the edge vector opposite
// the vertex over the triangle's area (area from the OperatorS record).
__global__ void vertex_curls_kernel(int64_t nv, const int32_t* __restrict__ v2t_beg,
                                    const int32_t* __restrict__ v2t_tri, const int8_t* __restrict__ v2t_loc,
                                    const double* __restrict__ V, const int32_t* __restrict__ T,
                                    const double* __restrict__ srec, double* q) {
    const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (v >= nv) return;
    for (int k = v2t_beg[v]; k < v2t_beg[v + 1]; ++k) {
        const int64_t t = v2t_tri[k];
        const d3 cb = edge_cb(V, T, t, v2t_loc[k]);
        const double A = srec[t * SREC + 12];
        q[3 * (int64_t)k + 0] = cb.x / A;
        q[3 * (int64_t)k + 1] = cb.y / A;
        q[3 * (int64_t)k + 2] = cb.z / A;
    }
}

void launch_prepare_vertex_curls(const DevGeom& g, cudaStream_t s) {
    if (g.nv == 0) return;
    vertex_curls_kernel<<<nblocks(g.nv, 128), 128, 0, s>>>(g.nv, g.v2t_beg, g.v2t_tri, g.v2t_loc, g.V, g.T, g.srec,
                                                            g.v2t_q);
    check_launch("vertex curls");
}

// N block (operatorN, operators.h: the hypersingular operator by the curl
// identity): N(v1, v2) = -f sum_{a ni v1} sum_{b ni v2} (q_a(v1) . q_b(v2)) S(a, b),
// f = 1/4 (1/2 on a vertex shared by both sides of a non-self block), in two
// contractions with the sparse curl matrices instead of 36 curl products per
// vertex pair:
//   1. U_k(x, v) = sum_{y ni v} q_y,k(v) S(x, y), k = x, y, z, for every
//      triangle x of one side and vertex v of the other (x is the side along
//      which S is contiguous in memory: coalesced reads, warp-uniform loops);
//   2. N(vx, v) = -f sum_{x ni vx} sum_k q_x,k(vx) U_k(x, v).
// S(a, b) (a on mesh 1, b on mesh 2) is the block of the matrix (lower
// storage at the triangles' positions) or a dense a-major temporary.
__device__ __forceinline__ double n_block_s(const double* __restrict__ hm_src, int64_t ld,
                                            const double* __restrict__ tmp, int64_t nt2, const int32_t* __restrict__ tpos,
                                            int64_t t1b, int64_t t2b, int64_t a, int64_t b) {
    return hm_src ? hm_src[lower_at(tpos[a], tpos[b], ld)] : tmp[(a - t1b) * nt2 + (b - t2b)];
}

__global__ void n_curl_s_kernel(int64_t txb, int64_t nx, int64_t vyb, int64_t nvy, int64_t tyb, int64_t tye,
                                int swap, const double* __restrict__ hm_src, int64_t ld, const double* __restrict__ tmp,
                                int64_t nt2, int64_t t1b, int64_t t2b, const int32_t* __restrict__ v2t_beg,
                                const int32_t* __restrict__ v2t_tri, const double* __restrict__ vq,
                                const int32_t* __restrict__ tpos, double* __restrict__ U) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= nx * nvy) return;
    const int64_t ix = idx % nx, iv = idx / nx;   // x fastest
    const int64_t x = txb + ix, v = vyb + iv;
    double u0 = 0.0, u1 = 0.0, u2 = 0.0;
    for (int k = v2t_beg[v]; k < v2t_beg[v + 1]; ++k) {
        const int64_t y = v2t_tri[k];
        if (y < tyb || y >= tye) continue;
        const double sv = swap ? n_block_s(hm_src, ld, tmp, nt2, tpos, t1b, t2b, y, x)
                               : n_block_s(hm_src, ld, tmp, nt2, tpos, t1b, t2b, x, y);
        u0 = fma(vq[3 * (int64_t)k], sv, u0);
        u1 = fma(vq[3 * (int64_t)k + 1], sv, u1);
        u2 = fma(vq[3 * (int64_t)k + 2], sv, u2);
    }
    double* Uv = U + iv * 3 * nx + ix;
    Uv[0] = u0;
    Uv[nx] = u1;
    Uv[2 * nx] = u2;
}

__global__ void n_curl_u_kernel(int64_t vxb, int64_t nvx, int64_t txb, int64_t txe, int64_t vyb, int64_t nvy, int same,
                                int swap, double coeff, const double* __restrict__ U, int64_t nx,
                                const int32_t* __restrict__ v2t_beg, const int32_t* __restrict__ v2t_tri,
                                const double* __restrict__ vq, int64_t nP, double* hm, int64_t ld, int rect) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= nvx * nvy) return;
    const int64_t jx = idx % nvx, jy = idx / nvx;   // vx fastest
    const int64_t i1 = swap ? jy : jx, i2 = swap ? jx : jy;
    if (same && i2 > i1) return;
    const int64_t vx = vxb + jx, vy = vyb + jy;
    const int64_t v1 = swap ? vy : vx, v2 = swap ? vx : vy;
    const double factor = same ? 0.25 : (v1 == v2 ? 0.5 : 0.25);
    const double* Uy = U + jy * 3 * nx;
    double r = 0.0;
    for (int k = v2t_beg[vx]; k < v2t_beg[vx + 1]; ++k) {
        const int64_t x = v2t_tri[k];
        if (x < txb || x >= txe) continue;
        const int64_t ix = x - txb;
        r = fma(vq[3 * (int64_t)k], Uy[ix], r);
        r = fma(vq[3 * (int64_t)k + 1], Uy[nx + ix], r);
        r = fma(vq[3 * (int64_t)k + 2], Uy[2 * nx + ix], r);
    }
    const double result = -factor * r;
    if (rect)   // rectangular output: row = v1's unknown, column = v2 within its range
        hm[(nP + v1) + i2 * ld] += result * coeff;
    else
        hm[lower_at(nP + v1, nP + v2, ld)] += result * coeff;
}

void launch_N_block(const DevGeom& g, int64_t v1b, int64_t v1e, int64_t t1b, int64_t t1e, int64_t v2b, int64_t v2e,
                    int64_t t2b, int64_t t2e, bool same, double coeff, const double* hm_src, int64_t ld,
                    const double* tmp, double* hm, cudaStream_t s, bool rect, bool s_contiguous_b) {
    const int64_t n1 = v1e - v1b, n2 = v2e - v2b;
    if (n1 <= 0 || n2 <= 0) return;
    ProfScope prof_("n_block", s);
    // x: the triangles along which S is contiguous (b for a dense temporary, the later mesh in the matrix)
    const int swap = s_contiguous_b ? 1 : 0;
    const int64_t txb = swap ? t2b : t1b, txe = swap ? t2e : t1e, nx = txe - txb;
    const int64_t vxb = swap ? v2b : v1b, nvx = swap ? n2 : n1;
    const int64_t vyb = swap ? v1b : v2b, nvy = swap ? n1 : n2;
    const int64_t tyb = swap ? t1b : t2b, tye = swap ? t1e : t2e;
    DevBuf U((size_t)nx * nvy * 3 * sizeof(double), s);
    n_curl_s_kernel<<<nblocks(nx * nvy, 256), 256, 0, s>>>(txb, nx, vyb, nvy, tyb, tye, swap, hm_src, ld, tmp,
                                                           t2e - t2b, t1b, t2b, g.v2t_beg, g.v2t_tri, g.v2t_q, g.tpos,
                                                           U.as<double>());
    check_launch("N block (S by curls)");
    n_curl_u_kernel<<<nblocks(nvx * nvy, 256), 256, 0, s>>>(vxb, nvx, txb, txe, vyb, nvy, same ? 1 : 0, swap, coeff,
                                                            U.as<double>(), nx, g.v2t_beg, g.v2t_tri, g.v2t_q, g.nP,
                                                            hm, ld, rect ? 1 : 0);
    check_launch("N block");
}

// ---------------------------------------------------------------------------
// Deflation (Details::deflate, assembleHeadMat.cpp:27-60): add M(i0,i0)/n to
// every vertex pair of each outermost mesh.  The coefficient is read by a
// separate launch so no thread can observe a partially deflated diagonal.
// ---------------------------------------------------------------------------
__global__ void deflate_coef_kernel(const double* hm, int64_t pos, int64_t ld, double inv_nb, double* coef) {
    coef[0] = hm[pos + pos * ld] * inv_nb;
}
__global__ void deflate_add_kernel(int64_t vb, int64_t n, int64_t nP, const double* coef, double* hm, int64_t ld) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= n * n) return;
    const int64_t i1 = idx % n, i2 = idx / n;
    if (i2 > i1) return;
    hm[(nP + vb + i1) + (nP + vb + i2) * ld] += coef[0];
}

void launch_deflate(const DevGeom& g, const std::vector<std::pair<int64_t, int64_t>>& vranges, int64_t i_first,
                    int64_t nb, double* hm, int64_t ld, double* scratch, cudaStream_t s) {
    ProfScope prof_("deflate", s);
    const int64_t pos = g.nP + i_first;
    deflate_coef_kernel<<<1, 1, 0, s>>>(hm, pos, ld, 1.0 / (double)nb, scratch);
    check_launch("deflate coef");
    for (const auto& r : vranges) {
        const int64_t n = r.second - r.first;
        deflate_add_kernel<<<nblocks(n * n, 256), 256, 0, s>>>(r.first, n, g.nP, scratch, hm, ld);
        check_launch("deflate add");
    }
}

// ---------------------------------------------------------------------------
// Internal lower-triangle matrix -> reference numbering, dense (both halves)
// or SymMatrix packed upper.  ipos(r) = r >= nv ? r - nv : r + nP.
// ---------------------------------------------------------------------------
__global__ void to_reference_dense_kernel(int64_t N, int64_t nv, int64_t nP, const double* __restrict__ hm,
                                          int64_t ld, double* out, int64_t ldo) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    for (int64_t j = blockIdx.y; j < N; j += gridDim.y) {
        const int64_t a = i >= nv ? i - nv : i + nP, b = j >= nv ? j - nv : j + nP;
        out[i + j * ldo] = hm[lower_at(a, b, ld)];
    }
}
__global__ void to_reference_packed_kernel(int64_t N, int64_t nv, int64_t nP, const double* __restrict__ hm,
                                           int64_t ld, double* out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    for (int64_t j = blockIdx.y; j < N; j += gridDim.y) {
        if (i > j) continue;
        const int64_t a = i >= nv ? i - nv : i + nP, b = j >= nv ? j - nv : j + nP;
        out[i + j * (j + 1) / 2] = hm[lower_at(a, b, ld)];
    }
}

void launch_symmetrize_to_reference(const DevGeom& g, const double* hm_int, int64_t ld_int, double* out,
                                    int64_t ld_out, bool packed, cudaStream_t s) {
    ProfScope prof_("to_reference", s);
    dim3 grid(nblocks(g.Nref, 256), (unsigned)std::min<int64_t>(g.Nref, 32768));
    if (packed)
        to_reference_packed_kernel<<<grid, 256, 0, s>>>(g.Nref, g.nv, g.nP, hm_int, ld_int, out);
    else
        to_reference_dense_kernel<<<grid, 256, 0, s>>>(g.Nref, g.nv, g.nP, hm_int, ld_int, out, ld_out);
    check_launch("to reference");
}

// Rows of an internal-numbered N_int x ncol block (column-major, ldi) to the
// reference numbering [vertices | triangle unknowns], Nref x ncol (ldo).
__global__ void rows_to_reference_kernel(int64_t Nref, int64_t nv, int64_t nP, int64_t ncol,
                                         const double* __restrict__ in, int64_t ldi, double* out, int64_t ldo) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= Nref) return;
    const int64_t a = r < nv ? nP + r : r - nv;
    for (int64_t c = blockIdx.y; c < ncol; c += gridDim.y) out[r + c * ldo] = in[a + c * ldi];
}

void launch_rows_to_reference(const DevGeom& g, int64_t ncol, const double* in, int64_t ldi, double* out, int64_t ldo,
                              cudaStream_t s) {
    if (ncol <= 0 || g.Nref <= 0) return;
    dim3 grid(nblocks(g.Nref, 256), (unsigned)std::min<int64_t>(ncol, 32768));
    rows_to_reference_kernel<<<grid, 256, 0, s>>>(g.Nref, g.nv, g.nP, ncol, in, ldi, out, ldo);
    check_launch("rows to reference");
}

// Reference-numbered dense (lower triangle read) -> internal lower triangle,
// identity on the padding.
__global__ void from_reference_dense_kernel(int64_t N, int64_t nv, int64_t nP, int64_t nPt,
                                            const double* __restrict__ in, int64_t ldi, double* hm, int64_t ld) {
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;   // internal row
    if (a >= N) return;
    for (int64_t b = blockIdx.y; b <= a; b += gridDim.y) {             // internal column
        const bool pa = (a >= nPt && a < nP), pb = (b >= nPt && b < nP);
        if (pa || pb) {
            hm[a + b * ld] = (a == b) ? 1.0 : 0.0;
            continue;
        }
        const int64_t i = a < nPt ? a + nv : a - nP, j = b < nPt ? b + nv : b - nP;
        hm[a + b * ld] = i >= j ? in[i + j * ldi] : in[j + i * ldi];
    }
}

__global__ void pad_identity_kernel(int64_t nPt, int64_t nP, double* hm, int64_t ld) {
    const int64_t a = nPt + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (a < nP) hm[a + a * ld] = 1.0;
}

void launch_pad_identity(const DevGeom& g, double* hm, int64_t ld, cudaStream_t s) {
    if (g.nP == g.nPt) return;
    ProfScope prof_("pad_identity", s);
    pad_identity_kernel<<<1, 128, 0, s>>>(g.nPt, g.nP, hm, ld);
    check_launch("pad identity");
}

void launch_from_reference_dense(const DevGeom& g, const double* in, int64_t ldi, double* hm, int64_t ld,
                                 cudaStream_t s) {
    ProfScope prof_("from_reference", s);
    dim3 grid(nblocks(g.N, 256), (unsigned)std::min<int64_t>(g.N, 32768));
    from_reference_dense_kernel<<<grid, 256, 0, s>>>(g.N, g.nv, g.nP, g.nPt, in, ldi, hm, ld);
    check_launch("from reference");
}

// ===========================================================================
// Mixed-precision HeadMat assembly
//
// Far pairs (centroid distance >= rho_far x the larger max edge) are computed
// by a 16 x 16 Gauss product rule in FP32 -- the same outer rule as the
// reference, with the analytic inner integral replaced by the rule on the
// other triangle.  Coordinates are taken relative to each triangle's centroid
// and the centroid difference is formed in FP64 before rounding, so the FP32
// distances carry no cancellation.  One pass over a triangle pair yields S,
// D(t1 -> vertices of t2) and D(t2 -> vertices of t1): the 256 point-point
// distances are shared.  Near pairs are appended to a list and recomputed
// with the FP64 analytic kernels.
// ===========================================================================
// floats per triangle: centroid (3 doubles), 16-point offsets, normal, h, area (double), 7-point offsets,
// area (FP32)
constexpr int GREC = kFarRecFloats, GREC_P7 = 64, GREC_AF = GREC_P7 + 21;
// The 16-point rule of c_rules[3] rounded to FP32 (weights, barycentric nodes).
__constant__ __align__(8) float c_w16[16] = {0.144315607677786f, 0.095091634267284f, 0.095091634267284f, 0.095091634267284f, 0.032458497623198f, 0.032458497623198f, 0.032458497623198f, 0.103217370534718f, 0.103217370534718f, 0.103217370534718f, 0.027230314174434f, 0.027230314174434f, 0.027230314174434f, 0.027230314174434f, 0.027230314174434f, 0.027230314174434f};
__constant__ float c_b16[16][3] = {
    {0.333333333333333f, 0.333333333333333f, 0.333333333333333f},
    {0.081414823414554f, 0.459292588292722f, 0.459292588292722f},
    {0.459292588292722f, 0.081414823414554f, 0.459292588292722f},
    {0.459292588292722f, 0.459292588292722f, 0.081414823414554f},
    {0.898905543365937f, 0.050547228317031f, 0.050547228317031f},
    {0.050547228317031f, 0.898905543365937f, 0.050547228317031f},
    {0.050547228317031f, 0.050547228317031f, 0.898905543365937f},
    {0.658861384496479f, 0.170569307751760f, 0.170569307751761f},
    {0.170569307751760f, 0.658861384496479f, 0.170569307751761f},
    {0.170569307751760f, 0.170569307751761f, 0.658861384496479f},
    {0.008394777409957f, 0.728492392955404f, 0.263112829634639f},
    {0.728492392955404f, 0.008394777409957f, 0.263112829634639f},
    {0.728492392955404f, 0.263112829634639f, 0.008394777409957f},
    {0.008394777409957f, 0.263112829634639f, 0.728492392955404f},
    {0.263112829634639f, 0.008394777409957f, 0.728492392955404f},
    {0.263112829634639f, 0.728492392955404f, 0.008394777409957f}};
// The 7-point rule of c_rules[2] rounded to FP32, for well-separated pairs; weights padded with a zero eighth
// lane (the packed pair (6, 6) counts point 6 once).
__constant__ __align__(8) float c_w7[8] = {0.2250f, 0.132394152788506f, 0.132394152788506f, 0.132394152788506f,
                                           0.125939180544828f, 0.125939180544828f, 0.125939180544828f, 0.f};
__constant__ float c_b7[7][3] = {{0.333333333333333f, 0.333333333333333f, 0.333333333333333f},
                                 {0.470142064105115f, 0.470142064105115f, 0.059715871789770f},
                                 {0.470142064105115f, 0.059715871789770f, 0.470142064105115f},
                                 {0.059715871789770f, 0.470142064105115f, 0.470142064105115f},
                                 {0.101286507323456f, 0.101286507323456f, 0.797426985353088f},
                                 {0.101286507323456f, 0.797426985353088f, 0.101286507323456f},
                                 {0.797426985353088f, 0.101286507323456f, 0.101286507323456f}};


__global__ void prepare_gg_kernel(int64_t nt, const double* __restrict__ V, const int32_t* __restrict__ T,
                                  float* grec) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const d3 p0 = dev::ld3(V + 3 * (int64_t)T[3 * t]);
    const d3 p1 = dev::ld3(V + 3 * (int64_t)T[3 * t + 1]);
    const d3 p2 = dev::ld3(V + 3 * (int64_t)T[3 * t + 2]);
    const d3 c = (p0 + p1 + p2) * (1.0 / 3.0);
    float* g = grec + t * GREC;
    double* gc = reinterpret_cast<double*>(g);
    gc[0] = c.x; gc[1] = c.y; gc[2] = c.z;
    for (int k = 0; k < 16; ++k) {
        const d3 v = bary_point(c_rules[3][k], p0, p1, p2) - c;
        g[6 + 3 * k] = (float)v.x; g[7 + 3 * k] = (float)v.y; g[8 + 3 * k] = (float)v.z;
    }
    const d3 nn = dev::cross(p1 - p0, p2 - p0);
    const double nrm = dev::norm(nn);
    g[54] = (float)(nn.x / nrm); g[55] = (float)(nn.y / nrm); g[56] = (float)(nn.z / nrm);
    g[57] = (float)fmax(dev::norm(p1 - p0), fmax(dev::norm(p2 - p1), dev::norm(p0 - p2)));
    reinterpret_cast<double*>(g + 58)[0] = 0.5 * nrm;
    g[60] = g[61] = g[62] = g[63] = 0.f;
    for (int k = 0; k < 7; ++k) {
        const d3 v = bary_point(c_rules[2][k], p0, p1, p2) - c;
        g[GREC_P7 + 3 * k] = (float)v.x; g[GREC_P7 + 3 * k + 1] = (float)v.y; g[GREC_P7 + 3 * k + 2] = (float)v.z;
    }
    g[GREC_AF] = (float)(0.5 * nrm);
    for (int k = GREC_AF + 1; k < GREC; ++k) g[k] = 0.f;
}

void launch_prepare_gg(const DevGeom& g, float* grec, cudaStream_t s) {
    ProfScope prof_("prepare_gg", s);
    prepare_gg_kernel<<<nblocks(g.nt, 128), 128, 0, s>>>(g.nt, g.V, g.T, grec);
    check_launch("prepare_gg");
}

// Packed FP32 pairs (two lanes per 64-bit register) and the sm_100-family
// FP32x2 instructions on them: one issue slot performs two FP32 operations.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float lo2(f2 x) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x));
    return a;
}
__device__ __forceinline__ float hi2(f2 x) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x));
    return b;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// 1/sqrt(x) as the single approximate instruction (about 2 ulp, like rsqrtf);
// flushing denormals is harmless here: x is a squared distance between
// points of separated triangles.
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

constexpr int FF_TI = 128, FF_TJ = 16;
constexpr float kFarTier7 = 36.f;   // squared: pairs at >= 6 max edges take the 7-point rule

// One thread per t1 row, looping over the CTA's FF_TJ staged t2 records.
__global__ void __launch_bounds__(FF_TI, 3) ff_block_kernel(const float* __restrict__ grec, int64_t t1b, int64_t n1,
                                                         int64_t t2b, int64_t n2, int same, int wantS, int wantD12,
                                                         int wantD21, double cS, const int32_t* __restrict__ tpos,
                                                         double* hm, int64_t ld, double* stmp, double* d12,
                                                         double* d21, int2* near, int* near_count, int near_cap,
                                                         float rho, int* err) {
    __shared__ __align__(16) float sJ[FF_TJ * GREC];
    __shared__ __align__(8) uint64_t bar;
    const int64_t i0 = (int64_t)blockIdx.y * FF_TI, j0 = (int64_t)blockIdx.x * FF_TJ;
    if (same && j0 + FF_TJ <= i0) return;
    const int nj = (int)(n2 - j0 < (int64_t)FF_TJ ? n2 - j0 : (int64_t)FF_TJ);
    if (!dev::stage_two(sJ, grec + (t2b + j0) * GREC, (uint32_t)(nj * GREC * 4), nullptr, nullptr, 0, &bar, err))
        return;
    const int64_t i = i0 + threadIdx.x;
    if (i >= n1) return;
    const float* g1 = grec + (t1b + i) * GREC;
    const double* c1p = reinterpret_cast<const double*>(g1);
    const double c1x = c1p[0], c1y = c1p[1], c1z = c1p[2];
    const f2* W = reinterpret_cast<const f2*>(c_w16);   // weight pairs, read from the constant bank
    // t1's 7 points, packed (0,1) (2,3) (4,5) (6,6) (the last pair's second lane has a zero weight), held
    // across the loop: most pairs take the 7-point rule
    f2 Px[4], Py[4], Pz[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float* p7 = g1 + GREC_P7;
        const int u = 2 * k, v = 2 * k + 1 < 7 ? 2 * k + 1 : 6;
        Px[k] = pk2(p7[3 * u], p7[3 * v]);
        Py[k] = pk2(p7[3 * u + 1], p7[3 * v + 1]);
        Pz[k] = pk2(p7[3 * u + 2], p7[3 * v + 2]);
    }
    const float n1x = g1[54], n1y = g1[55], n1z = g1[56], h1 = g1[57];
    const float A1f = g1[GREC_AF], cSf = (float)cS;
    for (int jj = 0; jj < nj; ++jj) {
        const int64_t j = j0 + jj;
        if (same && j < i) continue;
        const float* g2 = sJ + jj * GREC;
        const double* c2p = reinterpret_cast<const double*>(g2);
        // the centroid difference in FP64 (no cancellation), rounded once; the rest of the pair in FP32
        const float fx = (float)(c2p[0] - c1x), fy = (float)(c2p[1] - c1y), fz = (float)(c2p[2] - c1z);
        const float hmax = fmaxf(h1, g2[57]);
        const float dist2 = fmaf(fx, fx, fmaf(fy, fy, fz * fz));
        if (dist2 < rho * rho * hmax * hmax) {
            const int slot = atomicAdd(near_count, 1);
            if (slot < near_cap) near[slot] = make_int2((int)i, (int)j);
            continue;
        }
        const float n2x = g2[54], n2y = g2[55], n2z = g2[56];
        // r = d + Q_q - P_k (d: centroid difference, P_k / Q_q: the points' offsets in the planes of t1 / t2,
        // so P_k . n1 = Q_q . n2 = 0): r . n2 = d . n2 - P_k . n2 depends on k only and r . n1 = d . n1 + Q_q . n1
        // on q only, folded into the weights: WD[k] = w_k (r . n2), cq = -w_q (r . n1)
        const float dn2 = fmaf(fx, n2x, fmaf(fy, n2y, fz * n2z));
        const float dn1 = fmaf(fx, n1x, fmaf(fy, n1y, fz * n1z));
        const f2 DN2 = pk2(dn2, dn2), N2x = pk2(n2x, n2x), N2y = pk2(n2y, n2y), N2z = pk2(n2z, n2z);
        float s = 0.f, e0 = 0.f, e1 = 0.f, e2 = 0.f, u0 = 0.f, u1 = 0.f, u2 = 0.f;   // u: D21
        if (dist2 >= kFarTier7 * hmax * hmax) {
            // well separated (>= 6 max edges): the 7 x 7 product rule, within 1e-7 of the 16 x 16 one there
            const f2* W7 = reinterpret_cast<const f2*>(c_w7);
            f2 WD7[4], A7[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                WD7[k] = mul2(W7[k], sub2(DN2, fma2(Px[k], N2x, fma2(Py[k], N2y, mul2(Pz[k], N2z)))));
                A7[k] = pk2(0.f, 0.f);
            }
            const float* q7 = g2 + GREC_P7;
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                const float qx = q7[3 * q], qy = q7[3 * q + 1], qz = q7[3 * q + 2];
                const float wq = c_w7[q];
                const float cq = -wq * (dn1 + fmaf(qx, n1x, fmaf(qy, n1y, qz * n1z)));
                const f2 Yx = pk2(fx + qx, fx + qx), Yy = pk2(fy + qy, fy + qy), Yz = pk2(fz + qz, fz + qz),
                         CQ = pk2(cq, cq);
                f2 SQ = pk2(0.f, 0.f), K12 = pk2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const f2 rx = sub2(Yx, Px[k]), ry = sub2(Yy, Py[k]), rz = sub2(Yz, Pz[k]);
                    const f2 r2 = fma2(rx, rx, fma2(ry, ry, mul2(rz, rz)));
                    const f2 ir = pk2(rsqrt_ftz(lo2(r2)), rsqrt_ftz(hi2(r2)));
                    const f2 ir3 = mul2(mul2(ir, ir), ir);
                    SQ = fma2(W7[k], ir, SQ);
                    K12 = fma2(WD7[k], ir3, K12);
                    A7[k] = fma2(CQ, ir3, A7[k]);
                }
                s = fmaf(wq, lo2(SQ) + hi2(SQ), s);
                const float kq = wq * (lo2(K12) + hi2(K12));
                e0 = fmaf(kq, c_b7[q][0], e0);
                e1 = fmaf(kq, c_b7[q][1], e1);
                e2 = fmaf(kq, c_b7[q][2], e2);
            }
            if (wantD21 || (same && wantD12)) {
#pragma unroll
                for (int p = 0; p < 7; ++p) {
                    const float a = c_w7[p] * ((p & 1) ? hi2(A7[p / 2]) : lo2(A7[p / 2]));
                    u0 = fmaf(a, c_b7[p][0], u0);
                    u1 = fmaf(a, c_b7[p][1], u1);
                    u2 = fmaf(a, c_b7[p][2], u2);
                }
            }
        } else {
            // the 16 points of t1 in packed pairs (even p in the low lane, odd p in the high lane; the inner
            // products run two point pairs per FP32x2 instruction), loaded (L1) for the few pairs of this tier
            // instead of held across the loop: the registers go to more resident warps
            f2 P1x[8], P1y[8], P1z[8], WD[8], A21[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                P1x[k] = pk2(g1[6 + 6 * k], g1[9 + 6 * k]);
                P1y[k] = pk2(g1[7 + 6 * k], g1[10 + 6 * k]);
                P1z[k] = pk2(g1[8 + 6 * k], g1[11 + 6 * k]);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                WD[k] = mul2(W[k], sub2(DN2, fma2(P1x[k], N2x, fma2(P1y[k], N2y, mul2(P1z[k], N2z)))));
                A21[k] = pk2(0.f, 0.f);
            }
            for (int q = 0; q < 16; ++q) {
                const float qx = g2[6 + 3 * q], qy = g2[7 + 3 * q], qz = g2[8 + 3 * q];
                const float yx = fx + qx, yy = fy + qy, yz = fz + qz;
                const float wq = c_w16[q];
                const float cq = -wq * (dn1 + fmaf(qx, n1x, fmaf(qy, n1y, qz * n1z)));
                const f2 Yx = pk2(yx, yx), Yy = pk2(yy, yy), Yz = pk2(yz, yz), CQ = pk2(cq, cq);
                f2 SQ = pk2(0.f, 0.f), K12 = pk2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const f2 rx = sub2(Yx, P1x[k]), ry = sub2(Yy, P1y[k]), rz = sub2(Yz, P1z[k]);
                    const f2 r2 = fma2(rx, rx, fma2(ry, ry, mul2(rz, rz)));
                    const f2 ir = pk2(rsqrt_ftz(lo2(r2)), rsqrt_ftz(hi2(r2)));
                    const f2 ir3 = mul2(mul2(ir, ir), ir);
                    SQ = fma2(W[k], ir, SQ);
                    K12 = fma2(WD[k], ir3, K12);
                    A21[k] = fma2(CQ, ir3, A21[k]);
                }
                s = fmaf(wq, lo2(SQ) + hi2(SQ), s);
                const float kq = wq * (lo2(K12) + hi2(K12));
                e0 = fmaf(kq, c_b16[q][0], e0);
                e1 = fmaf(kq, c_b16[q][1], e1);
                e2 = fmaf(kq, c_b16[q][2], e2);
            }
            if (wantD21 || (same && wantD12)) {
#pragma unroll
                for (int p = 0; p < 16; ++p) {
                    const float a = c_w16[p] * ((p & 1) ? hi2(A21[p / 2]) : lo2(A21[p / 2]));
                    u0 = fmaf(a, c_b16[p][0], u0);
                    u1 = fmaf(a, c_b16[p][1], u1);
                    u2 = fmaf(a, c_b16[p][2], u2);
                }
            }
        }
        // the sums are FP32: scaled by the area product in FP32, widened once each
        const float AA = A1f * g2[GREC_AF];
        if (wantS) {
            if (hm)
                hm[lower_at(tpos[t1b + i], tpos[t2b + j], ld)] = (double)(s * (AA * cSf));
            else {
                stmp[i * n2 + j] = (double)(s * AA);
                if (same) stmp[j * n2 + i] = (double)(s * AA);
            }
        }
        if (wantD12) {
            double* o = d12 + (i * n2 + j) * 3;
            o[0] = (double)(e0 * AA); o[1] = (double)(e1 * AA); o[2] = (double)(e2 * AA);
        }
        if (wantD21 || (same && wantD12)) {
            double* o = same ? d12 + (j * n2 + i) * 3 : d21 + (j * n1 + i) * 3;
            o[0] = (double)(u0 * AA); o[1] = (double)(u1 * AA); o[2] = (double)(u2 * AA);
        }
    }
}

// OperatorS and, in out, the three P1 double-layer integrals of one triangle (OperatorS record p) at one point by the shared
// forms of the S / D tables: one logarithm per edge and one arctangent for both, h = r0.n, E_j = n.(r_j+1 x r_j+2).
template <bool WANT_S, bool WANT_D>
__device__ __forceinline__ double near_eval(const double* __restrict__ p, d3 x, double* out) {
    const d3 r0 = dev::ld3(p) - x, r1 = dev::ld3(p + 3) - x, r2 = dev::ld3(p + 6) - x, n = dev::ld3(p + 9);
    const double A2 = 2.0 * p[12], e0 = p[13], e1 = p[14], e2 = p[15];
    const double q0 = e0 * e0, q1 = e1 * e1, q2 = e2 * e2;
    const double d0 = fx::sqrt64(dev::dot(r0, r0)), d1 = fx::sqrt64(dev::dot(r1, r1)), d2 = fx::sqrt64(dev::dot(r2, r2));
    const double R0 = d0 + d1, R1 = d1 + d2, R2 = d2 + d0;
    const double l0 = fx::edge<false>(R0, e0, 0, 0, 0.0), l1 = fx::edge<false>(R1, e1, 0, 0, 0.0), l2 = fx::edge<false>(R2, e2, 0, 0, 0.0);
    const double m0 = l0 - l1, m2 = l2 - l1;
    const d3 nr = dev::cross(n, r0);
    const double E2 = dev::dot(nr, r1), E1 = -dev::dot(nr, r2);
    const double hh = 2.0 * dev::dot(r0, n), num = A2 * hh;
    const double den = fma(-4.0, d0 * d1 * d2, fma(d0, fma(R1, R1, -q1), fma(d1, fma(R2, R2, -q2), d2 * fma(R0, R0, -q0))));
    const double w = fx::half_angle<false>(num, den, 0, 0, 0.0);
    if (WANT_D) {
        out[0] = out[1] = out[2] = 0.0;
        if (!sd_flat2(hh)) {
            const double h4 = 0.25 * hh, iA = 2.0 * sd_rcp(A2), g02 = 0.5 * (q1 - q0 - q2);   // D0.D2
            out[1] = iA * fma(w, E1, h4 * fma(g02, m0, q2 * m2));
            out[2] = iA * fma(w, E2, h4 * fma(q0, m0, g02 * m2));
            out[0] = 2.0 * w - out[1] - out[2];
        }
    }
    if (!WANT_S) return 0.0;
    const double el = fma(A2, l1, fma(E2, m0, E1 * m2));
    return sd_flat2(num) ? el : fma(-hh, w, el);
}

// Near pairs: the FP64 analytic kernels of the reference (same outer rule).
// One lane per (pair, point of the rule): 16 lanes hold a pair, each lane
// evaluates the analytic integrals at its point (S and D21 over t1 at the
// points of t2, D12 over t2 at the points of t1, near_eval: one logarithm per
// edge, and it, the square roots and the arctangent on the integer pipe where
// their polynomials reach) and the weighted values are summed across the 16
// lanes by shuffles.  The 17926-unknown head's near pairs take 1.9 ms, with
// FP64 polynomials 3.9, with separate logarithms for S and D 5.2.  Short
// per-thread chains and many warps hide the latency of the
// FP64 transcendentals.
constexpr int NP_LANES = 16;

__global__ void __launch_bounds__(128) near_pairs_kernel(
    const int2* __restrict__ near, int count, const double* __restrict__ srec,
    const double* __restrict__ qrec, int64_t t1b, int64_t n1, int64_t t2b, int64_t n2, int same, int wantS,
    int wantD12, int wantD21, double cS, int order, const int32_t* __restrict__ tpos, double* hm, int64_t ld,
    double* stmp, double* d12, double* d21) {
    const int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / NP_LANES;   // pair
    const int m = threadIdx.x % NP_LANES;                                            // point of the rule
    const bool live = g < count;   // every lane takes part in the shuffles
    int64_t i = 0, j = 0;
    if (live) {
        i = near[g].x;
        j = near[g].y;
    }
    const int64_t a = t1b + i, b = t2b + j;
    const bool wantP = (wantD21 || (same && wantD12)) && !(same && i == j);
    double sv = 0.0, p[3] = {0, 0, 0}, e[3] = {0, 0, 0};
    if (live && m < c_nbpts[order]) {
        const double w = c_rules[order][m][3];
        if (wantS || wantP) {
            const d3 x2 = dev::ld3(qrec + b * QREC + 3 * m);
            double v[3] = {0, 0, 0};
            if (wantS && wantP)
                sv = w * near_eval<true, true>(srec + a * SREC, x2, v);
            else if (wantS)
                sv = w * near_eval<true, false>(srec + a * SREC, x2, v);
            else
                near_eval<false, true>(srec + a * SREC, x2, v);
            p[0] = w * v[0]; p[1] = w * v[1]; p[2] = w * v[2];
        }
        if (wantD12) {   // integral over t1 of P1SLP(t2)
            double v[3];
            near_eval<false, true>(srec + b * SREC, dev::ld3(qrec + a * QREC + 3 * m), v);
            e[0] = w * v[0]; e[1] = w * v[1]; e[2] = w * v[2];
        }
    }
    // Sums over the 16 lanes: each exchange halves the values a lane holds (8 additions a lane instead of 28 for seven
    // butterflies, in the same order); lane pair k of the group ends with value k.
    double r[8] = {sv, p[0], p[1], p[2], e[0], e[1], e[2], 0.0};
#pragma unroll
    for (int h = 4; h > 0; h >>= 1) {
        const bool up = m & (2 * h);
#pragma unroll
        for (int c = 0; c < h; ++c) {
            const double give = up ? r[c] : r[c + h];
            r[c] = (up ? r[c + h] : r[c]) + __shfl_xor_sync(0xffffffffu, give, 2 * h);
        }
    }
    const double v = r[0] + __shfl_xor_sync(0xffffffffu, r[0], 1);
    if (!live || (m & 1)) return;
    const int k = m / 2;
    if (k == 0) {
        if (!wantS) return;
        const double val = qrec[b * QREC + 48] * v;
        if (hm)
            hm[lower_at(tpos[a], tpos[b], ld)] = val * cS;
        else {
            stmp[i * n2 + j] = val;
            if (same) stmp[j * n2 + i] = val;
        }
    } else if (k < 4) {
        if (wantP) (same ? d12 + (j * n2 + i) * 3 : d21 + (j * n1 + i) * 3)[k - 1] = qrec[b * QREC + 48] * v;
    } else if (k < 7) {
        if (wantD12) d12[(i * n2 + j) * 3 + k - 4] = qrec[a * QREC + 48] * v;
    }
}

void launch_ff_block(const DevGeom& g, const float* grec, int64_t t1b, int64_t t1e, int64_t t2b, int64_t t2e,
                     bool same, bool wantS, bool wantD12, bool wantD21, double cS, double* hm, int64_t ld,
                     double* stmp, double* d12, double* d21, int2* near, int* near_count, int near_cap, float rho,
                     int* err, cudaStream_t s) {
    ProfScope prof_("ff_block", s);
    const int64_t n1 = t1e - t1b, n2 = t2e - t2b;
    dim3 grid(nblocks(n2, FF_TJ), nblocks(n1, FF_TI));
    ff_block_kernel<<<grid, FF_TI, 0, s>>>(grec, t1b, n1, t2b, n2, same ? 1 : 0, wantS ? 1 : 0, wantD12 ? 1 : 0,
                                           wantD21 ? 1 : 0, cS, g.tpos, hm, ld, stmp, d12, d21, near, near_count,
                                           near_cap, rho, err);
    check_launch("ff block");
}

void launch_near_pairs(const DevGeom& g, const int2* near, int count, int64_t t1b, int64_t t1e, int64_t t2b,
                       int64_t t2e, bool same, bool wantS, bool wantD12, bool wantD21, double cS, int order,
                       double* hm, int64_t ld, double* stmp, double* d12, double* d21, cudaStream_t s) {
    if (count <= 0) return;
    if (order < 0 || order > 3) throw Error(OMG_ERR_INVALID, "near pairs: rule of more than 16 points");
    ProfScope prof_("near_pairs", s);
    near_pairs_kernel<<<nblocks((int64_t)count * NP_LANES, 128), 128, 0, s>>>(near, count, g.srec, g.qrec,
                                                                              t1b, t1e - t1b, t2b,
                                                          t2e - t2b, same ? 1 : 0, wantS ? 1 : 0, wantD12 ? 1 : 0,
                                                          wantD21 ? 1 : 0, cS, order, g.tpos, hm, ld, stmp, d12, d21);
    check_launch("near pairs");
}

// ===========================================================================
// Sources and sensors
// ===========================================================================

// Interface::contains (OpenMEEG/src/interface.cpp:18-35) on an oriented solid angle.
__device__ __forceinline__ bool almost_eq(double x, double y) {
    return fabs(x - y) < 2.220446049250313e-16 * fabs(x + y) * 1e3 || fabs(x - y) < 2.2250738585072014e-308;
}
__device__ __forceinline__ bool interface_contains(double s) {
    const double fourpi = 12.566370614359172;
    if (almost_eq(s, -fourpi)) return true;
    if (almost_eq(s, 0.0)) return false;
    if (almost_eq(s, fourpi)) return true;
    return fabs(s) > 0.5 * fourpi;
}

// Mesh::solid_angle (mesh.cpp:239-244) of every mesh seen from every point:
// one CTA per point, a fixed-order tree reduction per mesh.
__global__ void mesh_solid_angles_kernel(const double* __restrict__ pts, int64_t pstride, int nmesh,
                                         const int64_t* __restrict__ tbeg, const double* __restrict__ srec,
                                         double* out) {
    __shared__ double red[256];
    const int64_t i = blockIdx.x;
    const d3 p = dev::ld3(pts + i * pstride);
    for (int m = 0; m < nmesh; ++m) {
        double acc = 0.0;
        for (int64_t t = tbeg[m] + threadIdx.x; t < tbeg[m + 1]; t += blockDim.x) {
            const double* s = srec + t * SREC;
            const d3 r0 = dev::ld3(s) - p, r1 = dev::ld3(s + 3) - p, r2 = dev::ld3(s + 6) - p;
            acc += dev::solid_angle(r0, r1, r2, dev::norm(r0), dev::norm(r1), dev::norm(r2), dev::ld3(s + 9), s[12]);
        }
        red[threadIdx.x] = acc;
        __syncthreads();
        for (int w = blockDim.x / 2; w > 0; w >>= 1) {
            if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
            __syncthreads();
        }
        if (threadIdx.x == 0) out[i * nmesh + m] = red[0];
        __syncthreads();
    }
}

// Same, screened in FP32 for the domain lookup: a closed mesh subtends 0 or
// +-4 pi, so only the classification |sum| > 2 pi matters.  The FP64 sum is
// taken where FP32 could tip that test:
//  * a triangle whose angle FP32 cannot be sure of.  With u = 2^-24 the errors
//    are at most 7 u 2A|r0| in num and 56 u d0 d1 d2 in den, together e below;
//    the angle is within 2% when |num| or den exceeds 100 e.  With den < 0 and a
//    smaller |num| (a point just off the triangle) even its sign is open, which
//    moves the sum by 4 pi.  FP64 drops the angle when |num| < 1e-10, so here
//    |num| has to be clear of that as well, or the angle below 2e-6 either way;
//  * a sum within 1 of 2 pi.
__global__ void mesh_solid_angles_screened_kernel(const double* __restrict__ pts, int64_t pstride, int nmesh,
                                                  const int64_t* __restrict__ tbeg, const double* __restrict__ srec,
                                                  double* out) {
    __shared__ float redf[256];
    __shared__ double red[256];
    const int64_t i = blockIdx.x;
    const d3 p = dev::ld3(pts + i * pstride);
    for (int m = 0; m < nmesh; ++m) {
        float acc = 0.f;
        bool doubt = false;
        for (int64_t t = tbeg[m] + threadIdx.x; t < tbeg[m + 1]; t += blockDim.x) {
            const double* s = srec + t * SREC;
            const float ax = (float)(s[0] - p.x), ay = (float)(s[1] - p.y), az = (float)(s[2] - p.z);
            const float bx = (float)(s[3] - p.x), by = (float)(s[4] - p.y), bz = (float)(s[5] - p.z);
            const float cx = (float)(s[6] - p.x), cy = (float)(s[7] - p.y), cz = (float)(s[8] - p.z);
            const float da = sqrtf(ax * ax + ay * ay + az * az), db = sqrtf(bx * bx + by * by + bz * bz),
                        dc = sqrtf(cx * cx + cy * cy + cz * cz);
            const float A2 = 2.f * (float)s[12], prod = da * db * dc;
            const float num = A2 * (ax * (float)s[9] + ay * (float)s[10] + az * (float)s[11]);
            const float den = prod + da * (bx * cx + by * cy + bz * cz) + db * (cx * ax + cy * ay + cz * az) +
                              dc * (ax * bx + ay * by + az * bz);
            const float e = 4e-6f * prod + 5e-7f * (A2 * da), mag = fabsf(num);
            if (mag > 1e-10f + 100.f * e || den > 1e-4f + 100.f * e)
                acc += 2.f * atan2f(num, den);
            else if (!(mag < 1e-10f - e))   // (so are infinities and NaN)
                doubt = true;
        }
        redf[threadIdx.x] = acc;
        doubt = __syncthreads_or(doubt);
        for (int w = blockDim.x / 2; w > 0; w >>= 1) {
            if (threadIdx.x < w) redf[threadIdx.x] += redf[threadIdx.x + w];
            __syncthreads();
        }
        const float sum = redf[0];
        __syncthreads();
        if (!doubt && fabsf(fabsf(sum) - 6.2831853f) > 1.f && sum == sum) {   // clear of the 2 pi boundary
            if (threadIdx.x == 0) out[i * nmesh + m] = fabsf(sum) < 6.2831853f ? 0.0 : (sum > 0 ? 1.0 : -1.0) *
                                                                                          12.566370614359172;
            continue;
        }
        double accd = 0.0;   // near the surface: the FP64 sum of the reference formula
        for (int64_t t = tbeg[m] + threadIdx.x; t < tbeg[m + 1]; t += blockDim.x) {
            const double* s = srec + t * SREC;
            const d3 r0 = dev::ld3(s) - p, r1 = dev::ld3(s + 3) - p, r2 = dev::ld3(s + 6) - p;
            accd += dev::solid_angle(r0, r1, r2, dev::norm(r0), dev::norm(r1), dev::norm(r2), dev::ld3(s + 9), s[12]);
        }
        red[threadIdx.x] = accd;
        __syncthreads();
        for (int w = blockDim.x / 2; w > 0; w >>= 1) {
            if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
            __syncthreads();
        }
        if (threadIdx.x == 0) out[i * nmesh + m] = red[0];
        __syncthreads();
    }
}

// Geometry::domain(point) (geometry.cpp:146-154, domain.cpp:12-17): the first
// domain all of whose boundaries agree with the point's inside/outside state.
// A boundary is an interface: the solid angles of its meshes are summed with
// their orientations (Interface::solid_angle, interface.cpp:40-45); the
// domain's per-mesh entries of one interface share a group index.
__global__ void domain_lookup_kernel(int64_t n, int nmesh, const double* __restrict__ sa, int ndom, int maxb,
                                     const int* __restrict__ dnb, const int* __restrict__ bmesh,
                                     const int* __restrict__ binside, const int* __restrict__ borient,
                                     const int* __restrict__ bgrp, int forced, int* dom, int* err) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (forced >= 0) {
        dom[i] = forced;
        return;
    }
    int found = -1;
    for (int d = 0; d < ndom && found < 0; ++d) {
        bool ok = true;
        double acc = 0.0;
        for (int k = 0; k < dnb[d]; ++k) {
            const int q = d * maxb + k;
            acc += borient[q] * sa[i * nmesh + bmesh[q]];
            if (k + 1 == dnb[d] || bgrp[q + 1] != bgrp[q]) {   // end of this interface's meshes
                if (interface_contains(acc) != (binside[q] != 0)) ok = false;
                acc = 0.0;
            }
        }
        if (ok) found = d;
    }
    dom[i] = found;
    if (found < 0) atomicExch(err, -1 /* OMG_ERR_INVALID: point in no domain */);
}

// Integrands of the DipSourceMat: Dipole::potential / Dipole::gradient
// (dipole.h:29-46) and the barycentric weights of PotentialDerivative
// (analytics.h:140-150, BarycentricCoordinates.h:33-69).
struct DsmTri {
    d3 p0, e10, e20, n;
    double d11, d12, d22;
};
__device__ __forceinline__ void subtriangle(d3& P0, d3& P1, d3& P2, int c) {
    const d3 m0 = (P1 + P2) * 0.5, m1 = (P2 + P0) * 0.5, m2 = (P0 + P1) * 0.5;
    if (c == 0) { P1 = m1; P2 = m2; }
    else if (c == 1) { P0 = m0; P2 = m2; }
    else if (c == 2) { P0 = m0; P1 = m1; }
    else { P0 = m0; P1 = m1; P2 = m2; }
}

constexpr int DSM_MAX_LEVELS = 12;
constexpr int DSM_STACK = 3 * (DSM_MAX_LEVELS + 1) + 4;
struct DsmNode {   // a triangle to refine: its corners, its own rule's values, the levels left
    double p[9], coarse[3], area;
    int level;
};

// Rule-weighted integrand values at one point (zero for k past the rule).
__device__ __forceinline__ void dsm_point(int kind, int order, const DsmTri& T, d3 r0, d3 q, double qn, const d3 P[3], int k,
                                          double acc[3]) {
    if (k >= c_nbpts[order]) return;
    const d3 r = bary_point(c_rules[order][k], P[0], P[1], P[2]);
    const double w = c_rules[order][k][3];
    const d3 x = r - r0;
    const double n2 = dev::dot(x, x), qx = dev::dot(q, x);
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(n2));
    const double e = fma(-(n2 * y), y, 1.0);   // (1 - e)^(-1/2) = 1 + e / 2 + 3 e^2 / 8: the binomial series
    y = fma(y * e, fma(0.375, e, 0.5), y);
    const double y2 = y * y, wy3 = w * (y2 * y);
    if (kind == 1) {
        acc[0] = fma(qx, wy3, acc[0]);
        return;
    }
    const double g = fma(-3.0 * dev::dot(T.n, x), qx * y2, qn) * wy3;
    const d3 v = r - T.p0;
    const double a1 = dev::dot(v, T.e10), a2 = dev::dot(v, T.e20);
    const double l1 = fma(T.d11, a1, T.d12 * a2), l2 = fma(T.d12, a1, T.d22 * a2);
    acc[0] = fma(g, 1.0 - l1 - l2, acc[0]);
    acc[1] = fma(g, l1, acc[1]);
    acc[2] = fma(g, l2, acc[2]);
}

// Integrator::integrate with adaptive_integration (integrator.h:44-48,228-252)
// by a warp, depth first with a stack in shared memory: eight lanes integrate
// each of a node's four children, two points a lane, so a node is about 150
// FP64 instructions deep (four lanes with 16 points each: 1800, which set the
// length of the deepest pairs' chains).  leaf(P, sub, ref) is called by every
// lane for each accepted node: its child P (corners), a child's area, the
// node's refined values.  levels > 0.
template <typename Leaf>
__device__ __forceinline__ void dsm_adaptive_warp(int kind, int order, int levels, double tol, const DsmTri& T, d3 r0,
                                                  d3 q, d3 R0, d3 R1, d3 R2, double area, DsmNode* st, int lane,
                                                  Leaf leaf) {
    const double qn = dev::dot(q, T.n);
    const int dim = kind == 0 ? 3 : 1;
    auto reduce = [&](double v[3], int width) {   // sum over groups of `width` lanes
        for (int o = width / 2; o > 0; o >>= 1)
            for (int k = 0; k < dim; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    };
    {
        double c[3] = {0.0, 0.0, 0.0};
        const d3 P[3] = {R0, R1, R2};
        dsm_point(kind, order, T, r0, q, qn, P, lane, c);
        reduce(c, 32);
        if (lane == 0) {
            for (int k = 0; k < 3; ++k) {
                st[0].p[3 * k] = P[k].x;
                st[0].p[3 * k + 1] = P[k].y;
                st[0].p[3 * k + 2] = P[k].z;
                st[0].coarse[k] = area * c[k];
            }
            st[0].area = area;
            st[0].level = levels;
        }
        __syncwarp();
    }
    const int child = lane >> 3, l8 = lane & 7;
    for (int sp = 1; sp > 0;) {
        --sp;
        d3 P[3] = {dev::ld3(st[sp].p), dev::ld3(st[sp].p + 3), dev::ld3(st[sp].p + 6)};
        const double c0 = st[sp].coarse[0], c1 = st[sp].coarse[1], c2 = st[sp].coarse[2], sub = 0.25 * st[sp].area;
        const int level = st[sp].level;
        __syncwarp();
        subtriangle(P[0], P[1], P[2], child);
        double mine[3] = {0.0, 0.0, 0.0};
        dsm_point(kind, order, T, r0, q, qn, P, l8, mine);
        dsm_point(kind, order, T, r0, q, qn, P, l8 + 8, mine);
        reduce(mine, 8);
        double ref[3] = {0.0, 0.0, 0.0};
        for (int k = 0; k < dim; ++k) {
            mine[k] *= sub;
            for (int c = 0; c < 4; ++c) ref[k] += __shfl_sync(0xffffffffu, mine[k], 8 * c);
        }
        double dn, cn;
        if (dim == 1) {
            dn = fabs(c0 - ref[0]);
            cn = fabs(c0);
        } else {
            const double e0 = c0 - ref[0], e1 = c1 - ref[1], e2 = c2 - ref[2];
            dn = sqrt(e0 * e0 + e1 * e1 + e2 * e2);
            cn = sqrt(c0 * c0 + c1 * c1 + c2 * c2);
        }
        if (dn <= tol * cn || level == 0) {   // (the same on every lane)
            leaf(P, sub, ref);
            continue;
        }
        if (l8 == 0) {   // child 0 on top
            DsmNode& n = st[sp + 3 - child];
            for (int k = 0; k < 3; ++k) {
                n.p[3 * k] = P[k].x;
                n.p[3 * k + 1] = P[k].y;
                n.p[3 * k + 2] = P[k].z;
                n.coarse[k] = mine[k];
            }
            n.area = sub;
            n.level = level - 1;
        }
        sp += 4;
        __syncwarp();
    }
}

// FP64: the first adaptive level of both integrands of every (dipole, triangle)
// pair, 80 points.  What depends on the triangle alone is tabled once per
// launch, by rule point (the triangle's 16 and each child's 16), lanes along
// the triangles: the point relative to the centroid c, the three P1 values (the
// first as the sum's difference from the others' had three times their error) and
// -3 n.(point - c).  With X = c - r0 (r0, q: the dipole) a point then takes 10
// FP64 operations for the potential and its three P1-weighted derivatives:
// r = X + (point - c), |r|^2, q.r, the reciprocal square root and its product with
// the weight run on the integer pipe beside them (fixed64.cuh), in 60-bit vectors
// with one exponent per pair.  Two separate adaptive integrations took ~110, on a
// pipe that bounds the DipSourceMat: 500 dipoles on 12960 triangles take 4.3 ms,
// with r and the products in FP64 (19 operations) 7.5, with the root as well (25) 9.8.
// A pair is settled here when |coarse - refined| <= tol |coarse| holds with a
// margin far above the rounding; the others (and those decided by rounding) are
// listed for dsm_fallback_kernel.
constexpr int DSM_FL = 7;   // table values per point

// FIXED: the point relative to c in block fixed point, its exponent per triangle in te.  Otherwise the point itself, so that
// point - r0 is rounded once.
template <bool FIXED>
__global__ void dsm_points_kernel(int64_t nt, const double* __restrict__ srec, int order, double* tab, int32_t* te) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const double* s = srec + t * SREC;
    const d3 R0 = dev::ld3(s), R1 = dev::ld3(s + 3), R2 = dev::ld3(s + 6), n = dev::ld3(s + 9);
    const d3 c = (R0 + R1 + R2) * (1.0 / 3.0);
    const d3 e10 = R1 - R0, e20 = R2 - R0;
    const double c11 = dev::dot(e10, e10), c12 = dev::dot(e10, e20), c22 = dev::dot(e20, e20);
    const double inv_det = 1.0 / (c11 * c22 - c12 * c12);
    const int np = c_nbpts[order];
    d3 P0 = R0, P1 = R1, P2 = R2;
    const int set = blockIdx.y;   // 0: the triangle; 1..4: its children
    int em = 0;
    for (const d3& R : {R0 - c, R1 - c, R2 - c})
        em = max(em, max((int)fx::expo(R.x), max((int)fx::expo(R.y), (int)fx::expo(R.z))));
    if (FIXED && set == 0) te[t] = em - 1022;
    if (set > 0) subtriangle(P0, P1, P2, set - 1);
    for (int k = 0; k < np; ++k) {
        const double* r = c_rules[order][k];
        const d3 x = bary_point(r, P0, P1, P2);
        const d3 d = x - c, v = x - R0;
        const double a1 = dev::dot(v, e10), a2 = dev::dot(v, e20);
        double* o = tab + (int64_t)(set * np + k) * DSM_FL * nt + t;
        if (FIXED) {   // (a rule's point is in the triangle, up to the digits of its barycentric coordinates)
            int64_t* f = reinterpret_cast<int64_t*>(o);
            f[0] = fx::fix60(d.x, max(em - (int)fx::expo(d.x), 0));
            f[nt] = fx::fix60(d.y, max(em - (int)fx::expo(d.y), 0));
            f[2 * nt] = fx::fix60(d.z, max(em - (int)fx::expo(d.z), 0));
        } else {
            o[0] = x.x;
            o[nt] = x.y;
            o[2 * nt] = x.z;
        }
        o[3 * nt] = inv_det * (c22 * a1 - c12 * a2);
        o[4 * nt] = inv_det * (c11 * a2 - c12 * a1);
        o[5 * nt] = -3.0 * dev::dot(n, d);   // (not 0: the rules' truncated digits do not sum to 1)
        o[6 * nt] = 1.0 - o[3 * nt] - o[4 * nt];
    }
}

// The tolerance at which a pair is settled by the first level: below tol by a margin that the rounding of the values (some
// 1e-15 of them) cannot turn.  Where there is none left (tol under 1e-14, or negative: always refine) the pairs are listed.
__device__ __forceinline__ double dsm_limit(double tol) { return tol * (1.0 - 1e-9) - 1e-14; }

// The dipole's part in block fixed point: X and q (limbs with 0 <= l < 2^30), the exponent E of X + (point - c), that of q,
// and how far the table's points shift.
struct DsmFix {
    int64_t X[3];
    int2 q[3];
    int E, qe, down;
    bool use;   // (finite, and far from the ends of the range)
};
__device__ __forceinline__ int2 dsm_limbs(int64_t i) { return make_int2((int)(i >> 30), (int)(i & 0x3FFFFFFF)); }
__device__ __forceinline__ DsmFix dsm_fix(d3 X, d3 q, int te) {
    DsmFix f;
    const int ex = (int)fx::expo(X.x), ey = (int)fx::expo(X.y), ez = (int)fx::expo(X.z);
    const int em = max(max(ex, max(ey, ez)), te + 1022) + 1;
    f.E = em - 1022;
    f.down = f.E - te;
    f.X[0] = fx::fix60(X.x, em - ex);
    f.X[1] = fx::fix60(X.y, em - ey);
    f.X[2] = fx::fix60(X.z, em - ez);
    const int qx = (int)fx::expo(q.x), qy = (int)fx::expo(q.y), qz = (int)fx::expo(q.z), qm = max(qx, max(qy, qz));
    f.q[0] = dsm_limbs(fx::fix60(q.x, qm - qx));
    f.q[1] = dsm_limbs(fx::fix60(q.y, qm - qy));
    f.q[2] = dsm_limbs(fx::fix60(q.z, qm - qz));
    f.qe = qm - 1022;
    f.use = abs(f.E) < 400 && qm > 100 && qm < 1900;   // (a moment of zero has no mantissa to cut)
    return f;
}

// One set of rule points: sums of w g (1, l1, l2) and w potential.  FIXED: r = X + (point - c), |r|^2 and q.r on the integer
// pipe; a point closer than 2^-6 of the pair's scale (and X or q that are not finite) in FP64.
template <bool FIXED>
__device__ __forceinline__ void dsm_set(const double* __restrict__ tab, int64_t nt, int order, d3 X, d3 q, double qn,
                                        double h3, const DsmFix& F, double acc[4]) {
    acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
    const int np = c_nbpts[order];
#pragma unroll 2
    for (int k = 0; k < np; ++k, tab += DSM_FL * nt) {
        const double w = c_rules[order][k][3];
        const uint64_t wm = fx::mant(w);
        const int we = (int)fx::expo(w);
        double qr, y, wy;
        bool exact = true;
        if (FIXED) {
            const int64_t* d = reinterpret_cast<const int64_t*>(tab);
            const int down = min(F.down, 63);
            const int2 r[3] = {dsm_limbs(F.X[0] + (d[0] >> down)), dsm_limbs(F.X[1] + (d[nt] >> down)),
                               dsm_limbs(F.X[2] + (d[2 * nt] >> down))};
            exact = !fx::rnorm60(r, F.E, wm, we, y, wy) || !F.use;
            const int64_t mid = (int64_t)F.q[0].x * r[0].y + (int64_t)F.q[0].y * r[0].x + (int64_t)F.q[1].x * r[1].y +
                                (int64_t)F.q[1].y * r[1].x + (int64_t)F.q[2].x * r[2].y + (int64_t)F.q[2].y * r[2].x;
            const int64_t hi = (int64_t)F.q[0].x * r[0].x + (int64_t)F.q[1].x * r[1].x + (int64_t)F.q[2].x * r[2].x;
            qr = fx::value60(hi + (mid >> 30), F.qe + F.E);
        }
        if (!FIXED || __any_sync(__activemask(), exact)) {
            double dx = tab[0], dy = tab[nt], dz = tab[2 * nt];
            if (FIXED) {
                const int te = F.E - F.down;
                dx = fx::value60(__double_as_longlong(dx), te);
                dy = fx::value60(__double_as_longlong(dy), te);
                dz = fx::value60(__double_as_longlong(dz), te);
            }
            const double rx = X.x + dx, ry = X.y + dy, rz = X.z + dz;
            const double n2 = fma(rx, rx, fma(ry, ry, rz * rz));
            const double qr1 = fma(q.x, rx, fma(q.y, ry, q.z * rz));
            double wy1;
            const double y1 = fx::rsqrt64(n2, wm, we, w, wy1);
            if (exact) {
                qr = qr1;
                y = y1;
                wy = wy1;
            }
        }
        const double y2 = y * y, wy3 = y2 * wy;
        acc[3] = fma(qr, wy3, acc[3]);
        const double g = fma(h3 + tab[5 * nt], qr * y2, qn) * wy3;   // w (q.n - 3 (q.r) (n.r) / r^2) / r^3
        acc[0] = fma(tab[6 * nt], g, acc[0]);
        acc[1] = fma(tab[3 * nt], g, acc[1]);
        acc[2] = fma(tab[4 * nt], g, acc[2]);
    }
}

// Mixed precision: the first adaptive level in FP32 with coordinates relative
// to the triangle centroid.  The FP32 value is kept only when the acceptance
// test |coarse - refined| <= tol |coarse| (integrator.h:245) holds with a
// factor-2 margin -- a decision FP32 rounding cannot flip; otherwise the
// caller recomputes in FP64.
struct DsmTriF {
    float3 p0, e10, e20, n;   // p0 relative to the centroid
    float d11, d12, d22;
};
__device__ __forceinline__ float3 fmid(float3 a, float3 b) {
    return make_float3(0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z));
}
// Both integrands of the first level at once, sharing the point's distance:
// out[0..2] the kind-0 values (P1-weighted normal derivative), out[3] the
// kind-1 value (potential); the expressions of the separate evaluations.
__device__ __forceinline__ void dsm_eval2_f(const DsmTriF& T, float3 xc, float3 q, float3 v, float out[4]) {
    const float3 x = make_float3(xc.x + v.x, xc.y + v.y, xc.z + v.z);   // r - r0
    const float n2 = x.x * x.x + x.y * x.y + x.z * x.z;
    const float qx = q.x * x.x + q.y * x.y + q.z * x.z;
    out[3] = qx / (n2 * sqrtf(n2));
    const float inv = 1.f / n2;
    const float3 g = make_float3(q.x - 3.f * qx * x.x * inv, q.y - 3.f * qx * x.y * inv, q.z - 3.f * qx * x.z * inv);
    const float gn = (g.x * T.n.x + g.y * T.n.y + g.z * T.n.z) * (inv * sqrtf(inv));
    const float3 w = make_float3(v.x - T.p0.x, v.y - T.p0.y, v.z - T.p0.z);   // r - p0
    const float a1 = w.x * T.e10.x + w.y * T.e10.y + w.z * T.e10.z;
    const float a2 = w.x * T.e20.x + w.y * T.e20.y + w.z * T.e20.z;
    const float l1 = T.d11 * a1 + T.d12 * a2, l2 = T.d12 * a1 + T.d22 * a2;
    out[0] = gn * (1.f - l1 - l2);
    out[1] = gn * l1;
    out[2] = gn * l2;
}
__device__ __forceinline__ void dsm_rule2_f(const DsmTriF& T, float3 xc, float3 q, float3 P0, float3 P1, float3 P2,
                                            float area, float res[4]) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int k = 0; k < 16; ++k) {
        const float b0 = c_b16[k][0], b1 = c_b16[k][1], b2 = c_b16[k][2];
        const float3 v = make_float3(b0 * P0.x + b1 * P1.x + b2 * P2.x, b0 * P0.y + b1 * P1.y + b2 * P2.y,
                                     b0 * P0.z + b1 * P1.z + b2 * P2.z);
        float e[4];
        dsm_eval2_f(T, xc, q, v, e);
        const float w = c_w16[k];
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] = fmaf(w, e[c], acc[c]);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) res[c] = area * acc[c];
}
// The first adaptive level of both integrals in one pass over the 80 points
// (the 16-point rule on the triangle and on its four halves-of-edges
// subtriangles): okv / okp tell whether FP32 settles the kind-0 (v, three
// values) / kind-1 (p) integral, i.e. |coarse - refined| <= tol |coarse| / 2;
// v and p are then the refined values.
__device__ void dsm_first_level2_f32(double tol, const DsmTriF& T, float3 xc, float3 q, float3 R0, float3 R1,
                                     float3 R2, float area, double v[3], double p[1], bool& okv, bool& okp) {
    float coarse[4];
    dsm_rule2_f(T, xc, q, R0, R1, R2, area, coarse);
    const float3 m0 = fmid(R1, R2), m1 = fmid(R2, R0), m2 = fmid(R0, R1);
    const float sub = 0.25f * area;
    float a[4], b[4], c[4], d[4];
    dsm_rule2_f(T, xc, q, R0, m1, m2, sub, a);
    dsm_rule2_f(T, xc, q, m0, R1, m2, sub, b);
    dsm_rule2_f(T, xc, q, m0, m1, R2, sub, c);
    dsm_rule2_f(T, xc, q, m0, m1, m2, sub, d);
    // the sums and the test in FP32 (GB300's FP64 pipe runs at 1/64 of the FP32 rate): their rounding,
    // ~1e-7 of |coarse|, is far inside the factor-2 margin of the test (tol / 2 = 5e-4 of |coarse|)
    float ref[4], dnv = 0.f, cnv = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) ref[k] = (a[k] + b[k]) + (c[k] + d[k]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float e = coarse[k] - ref[k];
        dnv = fmaf(e, e, dnv);
        cnv = fmaf(coarse[k], coarse[k], cnv);
    }
    const float ht = 0.5f * (float)tol;
    okv = dnv <= ht * ht * cnv;
    okp = fabsf(coarse[3] - ref[3]) <= ht * fabsf(coarse[3]);
    for (int k = 0; k < 3; ++k) v[k] = ref[k];
    p[0] = ref[3];
}

// FP32 first-level record of a triangle (coordinates relative to its
// centroid, kept in FP64), built once per DipSourceMat launch.
struct DsmRecF {
    DsmTriF T;
    float3 F1, F2;   // vertices 1 and 2 relative to the centroid (vertex 0 is T.p0)
    float area;
    double cx, cy, cz;
};

__global__ void dsm_prepare_f_kernel(int64_t nt, const double* __restrict__ srec, DsmRecF* rec) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const double* s = srec + t * SREC;
    const d3 R0 = dev::ld3(s), R1 = dev::ld3(s + 3), R2 = dev::ld3(s + 6), n = dev::ld3(s + 9);
    const d3 e10 = R1 - R0, e20 = R2 - R0;
    const double c11 = dev::dot(e10, e10), c12 = dev::dot(e10, e20), c22 = dev::dot(e20, e20);
    const double inv_det = 1.0 / (c11 * c22 - c12 * c12);
    const d3 c = (R0 + R1 + R2) * (1.0 / 3.0);
    const d3 a0 = R0 - c, a1 = R1 - c, a2 = R2 - c;
    DsmRecF r;
    r.T.p0 = make_float3((float)a0.x, (float)a0.y, (float)a0.z);
    r.T.n = make_float3((float)n.x, (float)n.y, (float)n.z);
    r.T.e10 = make_float3((float)e10.x, (float)e10.y, (float)e10.z);
    r.T.e20 = make_float3((float)e20.x, (float)e20.y, (float)e20.z);
    r.T.d11 = (float)(c22 * inv_det);
    r.T.d12 = (float)(-c12 * inv_det);
    r.T.d22 = (float)(c11 * inv_det);
    r.F1 = make_float3((float)a1.x, (float)a1.y, (float)a1.z);
    r.F2 = make_float3((float)a2.x, (float)a2.y, (float)a2.z);
    r.area = (float)s[12];
    r.cx = c.x;
    r.cy = c.y;
    r.cz = c.z;
    rec[t] = r;
}

// Pair (dipole i, triangle t) of the DipSourceMat: the triangle's geometry
// for the integrator and the boundary coefficient, or false when the pair
// contributes nothing (dipole in no domain or a zero-conductivity one,
// triangle not on a boundary of the dipole's domain).
struct DsmPair {
    DsmTri T;
    d3 r0, q, R0, R1, R2;
    double area, coeffD, sigma;
    int m;
};

// The boundary coefficient of the pair, or false when it contributes nothing.
__device__ __forceinline__ bool dsm_pair_coeff(int64_t i, int64_t t, const int32_t* __restrict__ tmesh,
                                               const int* __restrict__ orient, const int* __restrict__ dom, int maxb,
                                               const int* __restrict__ dnb, const int* __restrict__ bmesh,
                                               const int* __restrict__ binside, const double* __restrict__ dsigma,
                                               DsmPair& P) {
    const int d = dom[i];
    if (d < 0) return false;
    P.sigma = dsigma[d];
    if (P.sigma == 0.0) return false;
    P.m = tmesh[t];
    bool on = false;
    for (int k = 0; k < dnb[d]; ++k)
        if (bmesh[d * maxb + k] == P.m) {
            P.coeffD = (binside[d * maxb + k] ? -kK : kK) * orient[d * maxb + k];
            on = true;
        }
    return on;
}

__device__ __forceinline__ bool dsm_pair(int64_t i, int64_t t, const double* __restrict__ dip,
                                         const double* __restrict__ srec, const int32_t* __restrict__ tmesh,
                                         const int* __restrict__ orient, const int* __restrict__ dom, int maxb,
                                         const int* __restrict__ dnb, const int* __restrict__ bmesh,
                                         const int* __restrict__ binside, const double* __restrict__ dsigma,
                                         DsmPair& P) {
    if (!dsm_pair_coeff(i, t, tmesh, orient, dom, maxb, dnb, bmesh, binside, dsigma, P)) return false;
    const double* s = srec + t * SREC;
    P.R0 = dev::ld3(s);
    P.R1 = dev::ld3(s + 3);
    P.R2 = dev::ld3(s + 6);
    P.T.p0 = P.R0;
    P.T.n = dev::ld3(s + 9);
    P.T.e10 = P.R1 - P.R0;
    P.T.e20 = P.R2 - P.R0;
    const double c11 = dev::dot(P.T.e10, P.T.e10), c12 = dev::dot(P.T.e10, P.T.e20),
                 c22 = dev::dot(P.T.e20, P.T.e20);
    const double inv_det = 1.0 / (c11 * c22 - c12 * c12);
    P.T.d11 = c22 * inv_det;
    P.T.d12 = -c12 * inv_det;
    P.T.d22 = c11 * inv_det;
    P.r0 = dev::ld3(dip + 6 * i);
    P.q = dev::ld3(dip + 6 * i + 3);
    P.area = s[12];
    return true;
}

// SourceMatrix<Dipole> (assembleSourceMat.cpp:66-104) with
// operatorPotentialDerivative / operatorPotential (operators.cpp:40-88):
// one thread per (dipole, triangle).  P0 rows are written directly (one
// triangle per row); the three P1 contributions go to `p1tmp` for a
// fixed-order vertex gather (the reference accumulates them atomically).
// A pair whose first adaptive level settles (FP64, or FP32 in mixed precision)
// is written here; the others are listed (with which of the two integrals is
// left) for the FP64 adaptive integration in dsm_fallback_kernel, so the warps
// of that deep recursion are not held up by pairs that need none.
constexpr int DSM_T_BITS = 29;   // triangle index bits of a list entry; the two top bits: integrals left

__global__ void dsm_kernel(int64_t dip0, int64_t ndc, const double* __restrict__ dip, int64_t nt,
                           const double* __restrict__ srec, const int32_t* __restrict__ tmesh,
                           const int64_t* __restrict__ tidx_ref, const int* __restrict__ barrier,
                           const int* __restrict__ orient, const int* __restrict__ dom, int maxb,
                           const int* __restrict__ dnb, const int* __restrict__ bmesh,
                           const int* __restrict__ binside, const double* __restrict__ dsigma, int order, int levels,
                           double tol, int64_t nv, int perm, double* out, int64_t ldo, double* p1tmp,
                           const double* __restrict__ tab, const int32_t* __restrict__ te, int2* left, int* nleft) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t il = blockIdx.y;
    if (t >= nt || il >= ndc) return;
    const int64_t i = dip0 + il;
    double* o3 = p1tmp + (il * nt + t) * 3;
    DsmPair P;
    if (!dsm_pair_coeff(i, t, tmesh, orient, dom, maxb, dnb, bmesh, binside, dsigma, P)) {
        o3[0] = o3[1] = o3[2] = 0.0;
        return;
    }
    const bool p0row = !barrier[P.m];
    const double* s = srec + t * SREC;
    const d3 n = dev::ld3(s + 9), q = dev::ld3(dip + 6 * i + 3);
    const d3 X = (dev::ld3(s) + dev::ld3(s + 3) + dev::ld3(s + 6)) * (1.0 / 3.0) - dev::ld3(dip + 6 * i);
    const double qn = dev::dot(q, n), h3 = -3.0 * dev::dot(n, X), area = s[12];
    const int64_t set = (int64_t)c_nbpts[order] * DSM_FL * nt;
    double v[4];
    const DsmFix F = dsm_fix(X, q, te[t]);
    dsm_set<true>(tab + t, nt, order, X, q, qn, h3, F, v);
    bool okv = true, okp = true;
    if (levels == 0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] *= area;
    } else {
        double ref[4] = {0.0, 0.0, 0.0, 0.0};
        for (int c = 1; c <= 4; ++c) {
            double a[4];
            dsm_set<true>(tab + c * set + t, nt, order, X, q, qn, h3, F, a);
#pragma unroll
            for (int k = 0; k < 4; ++k) ref[k] = fma(0.25 * area, a[k], ref[k]);
        }
        const double lim = dsm_limit(tol);
        double d2 = 0.0, c2 = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] *= area;
            const double e = v[k] - ref[k];
            if (k < 3) {
                d2 = fma(e, e, d2);
                c2 = fma(v[k], v[k], c2);
            } else {
                okp = lim >= 0.0 && fabs(e) <= lim * fabs(v[k]);
            }
        }
        okv = lim >= 0.0 && d2 <= lim * lim * c2;
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = ref[k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) o3[k] = okv ? v[k] * P.coeffD : 0.0;
    if (p0row && okp) {
        const int64_t ref = tidx_ref[t];
        out[(perm ? ref - nv : ref) + i * ldo] = v[3] * (P.coeffD / P.sigma);
    }
    const int need = (okv ? 0 : 1) | (p0row && !okp ? 2 : 0);
    if (need) left[atomicAdd(nleft, 1)] = make_int2((int)il, (int)t | (need << DSM_T_BITS));
}

// Mixed precision: the first level in FP32 (the 16-point rule, levels > 0).
__global__ void dsm_mixed_kernel(int64_t dip0, int64_t ndc, const double* __restrict__ dip, int64_t nt,
                                 const int32_t* __restrict__ tmesh, const int64_t* __restrict__ tidx_ref,
                                 const int* __restrict__ barrier, const int* __restrict__ orient,
                                 const int* __restrict__ dom, int maxb, const int* __restrict__ dnb,
                                 const int* __restrict__ bmesh, const int* __restrict__ binside,
                                 const double* __restrict__ dsigma, double tol, int64_t nv, int perm, double* out,
                                 int64_t ldo, double* p1tmp, const DsmRecF* __restrict__ recf, int2* left, int* nleft) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t il = blockIdx.y;
    if (t >= nt || il >= ndc) return;
    const int64_t i = dip0 + il;
    double* o3 = p1tmp + (il * nt + t) * 3;
    o3[0] = o3[1] = o3[2] = 0.0;
    DsmPair P;
    const int64_t ref = tidx_ref[t];
    const int64_t row = perm ? ref - nv : ref;
    if (!dsm_pair_coeff(i, t, tmesh, orient, dom, maxb, dnb, bmesh, binside, dsigma, P)) return;
    const bool p0row = !barrier[P.m];
    const DsmRecF R = recf[t];
    const double* dp = dip + 6 * i;
    const float3 xc = make_float3((float)(R.cx - dp[0]), (float)(R.cy - dp[1]), (float)(R.cz - dp[2]));
    const float3 qf = make_float3((float)dp[3], (float)dp[4], (float)dp[5]);
    double v[3], pf[1];
    bool f32v, f32p;
    dsm_first_level2_f32(tol, R.T, xc, qf, R.T.p0, R.F1, R.F2, R.area, v, pf, f32v, f32p);
    f32p = f32p && p0row;
    // FP32-accurate values: scaled in FP32 (an FP64 division per pair costs more than the pair's
    // FP32 work on GB300)
    const float cf = (float)P.coeffD;
    if (f32v) {
        o3[0] = (double)((float)v[0] * cf);
        o3[1] = (double)((float)v[1] * cf);
        o3[2] = (double)((float)v[2] * cf);
    }
    if (f32p) out[row + i * ldo] = (double)((float)pf[0] * (cf / (float)P.sigma));
    const int need = (f32v ? 0 : 1) | (p0row && !f32p ? 2 : 0);
    if (need) left[atomicAdd(nleft, 1)] = make_int2((int)il, (int)t | (need << DSM_T_BITS));
}

// The listed pairs of the first pass: FP64 adaptive integration of the
// integrals it did not settle (a warp per pair, grid-stride over the
// device-side count).  A walk is a serial chain of nodes, so what bounds it is
// the latency of one node: eight lanes per child and two points a lane (of 16)
// instead of a lane per child.  The FP64 source matrix of 8 dipoles on 960
// triangles took 0.21 ms after 0.58 with four lanes a pair.
constexpr int DSM_WARPS = 4;
__global__ void __launch_bounds__(32 * DSM_WARPS) dsm_fallback_kernel(
    int64_t dip0, int64_t nt, const double* __restrict__ dip, const double* __restrict__ srec,
    const int32_t* __restrict__ tmesh, const int64_t* __restrict__ tidx_ref, const int* __restrict__ orient,
    const int* __restrict__ dom, int maxb, const int* __restrict__ dnb, const int* __restrict__ bmesh,
    const int* __restrict__ binside, const double* __restrict__ dsigma, int order, int levels, double tol, int64_t nv,
    int perm, double* out, int64_t ldo, double* p1tmp, const int2* __restrict__ left, const int* __restrict__ nleft) {
    __shared__ DsmNode stack[DSM_WARPS][DSM_STACK];
    const int n = *nleft;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int idx = blockIdx.x * DSM_WARPS + warp; idx < n; idx += gridDim.x * DSM_WARPS) {
        const int2 e = left[idx];
        const int64_t il = e.x, t = e.y & ((1 << DSM_T_BITS) - 1);
        const int need = (int)((unsigned)e.y >> DSM_T_BITS);
        const int64_t i = dip0 + il;
        DsmPair P;
        if (!dsm_pair(i, t, dip, srec, tmesh, orient, dom, maxb, dnb, bmesh, binside, dsigma, P)) continue;
        double v[3] = {0.0, 0.0, 0.0};
        auto add = [&](const d3*, double, const double* ref) {
            for (int k = 0; k < 3; ++k) v[k] += ref[k];
        };
        if (need & 1) {
            dsm_adaptive_warp(0, order, levels, tol, P.T, P.r0, P.q, P.R0, P.R1, P.R2, P.area, stack[warp], lane, add);
            if (lane == 0) {
                double* o3 = p1tmp + (il * nt + t) * 3;
                o3[0] = v[0] * P.coeffD;
                o3[1] = v[1] * P.coeffD;
                o3[2] = v[2] * P.coeffD;
            }
        }
        if (need & 2) {
            v[0] = 0.0;
            dsm_adaptive_warp(1, order, levels, tol, P.T, P.r0, P.q, P.R0, P.R1, P.R2, P.area, stack[warp], lane, add);
            const int64_t ref = tidx_ref[t];
            if (lane == 0) out[(perm ? ref - nv : ref) + i * ldo] = v[0] * (P.coeffD / P.sigma);
        }
    }
}

__global__ void dsm_gather_kernel(int64_t dip0, int64_t ndc, int64_t nv, int64_t nt, const double* __restrict__ p1tmp,
                                  const int32_t* __restrict__ v2t_beg, const int32_t* __restrict__ v2t_tri,
                                  const int8_t* __restrict__ v2t_loc, int64_t nP, int perm, double* out,
                                  int64_t ldo) {
    const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t il = blockIdx.y;
    if (v >= nv || il >= ndc) return;
    double sum = 0.0;
    bool any = false;
    for (int k = v2t_beg[v]; k < v2t_beg[v + 1]; ++k) {
        const double x = p1tmp[(il * nt + v2t_tri[k]) * 3 + v2t_loc[k]];
        if (x != 0.0) any = true;
        sum += x;
    }
    if (any) out[(perm ? nP + v : v) + (dip0 + il) * ldo] = sum;
}

// Danielsson's point-triangle distance (danielsson.cpp:26-74) with every
// operation rounded separately, in the reference's order (Vect3 dotprod and
// norm, vect3.h:72-73,111): no contraction into fused multiply-adds, so the
// distances equal the reference's double-precision ones bit for bit.  A point
// above an edge shared by two triangles is mathematically equidistant from
// both; which one is "nearest" is decided by the rounding of these
// operations, and EITSourceMat injects current into that triangle (and
// Head2EEGMat, with several interfaces, pairs it with another's weights).
__device__ __forceinline__ double dot_rn(d3 a, d3 b) {
    return __dadd_rn(__dadd_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)), __dmul_rn(a.z, b.z));
}
__device__ __forceinline__ d3 sub_rn(d3 a, d3 b) {
    return {__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y), __dsub_rn(a.z, b.z)};
}
__device__ double danielsson_rn(d3 p, const d3 P[3], double al[3]) {
    int idx[3] = {0, 1, 2};
    int nb = 3;
    al[0] = al[1] = al[2] = 0.0;
    for (;;) {
        if (nb == 1) {
            al[idx[0]] = 1.0;
            const d3 d = sub_rn(p, P[idx[0]]);
            return __dsqrt_rn(dot_rn(d, d));
        }
        d3 A0Ai[3];
        for (int i = 1; i < nb; ++i) A0Ai[i] = sub_rn(P[idx[i]], P[idx[0]]);
        const d3 A0M = sub_rn(p, P[idx[0]]);
        if (nb == 2) {
            al[idx[1]] = __ddiv_rn(dot_rn(A0M, A0Ai[1]), dot_rn(A0Ai[1], A0Ai[1]));
            al[idx[0]] = __dsub_rn(1.0, al[idx[1]]);
        } else {
            const double a00 = dot_rn(A0Ai[1], A0Ai[1]), a10 = dot_rn(A0Ai[1], A0Ai[2]),
                         a11 = dot_rn(A0Ai[2], A0Ai[2]);
            const double b0 = dot_rn(A0M, A0Ai[1]), b1 = dot_rn(A0M, A0Ai[2]);
            const double dd = __dsub_rn(__dmul_rn(a00, a11), __dmul_rn(a10, a10));
            al[idx[1]] = __ddiv_rn(__dsub_rn(__dmul_rn(b0, a11), __dmul_rn(b1, a10)), dd);
            al[idx[2]] = __ddiv_rn(__dsub_rn(__dmul_rn(a00, b1), __dmul_rn(a10, b0)), dd);
            al[idx[0]] = __dsub_rn(__dsub_rn(1.0, al[idx[1]]), al[idx[2]]);
        }
        int neg = -1;
        for (int i = 0; i < nb; ++i)
            if (al[idx[i]] < 0) {
                neg = i;
                break;
            }
        if (neg >= 0) {
            al[idx[neg]] = 0;
            const int tmp = idx[neg];
            idx[neg] = idx[nb - 1];
            idx[nb - 1] = tmp;
            --nb;
            continue;
        }
        d3 MH = {-A0M.x, -A0M.y, -A0M.z};
        for (int i = 1; i < nb; ++i) {
            const double a = al[idx[i]];
            MH = {__dadd_rn(MH.x, __dmul_rn(a, A0Ai[i].x)), __dadd_rn(MH.y, __dmul_rn(a, A0Ai[i].y)),
                  __dadd_rn(MH.z, __dmul_rn(a, A0Ai[i].z))};
        }
        return __dsqrt_rn(dot_rn(MH, MH));
    }
}

// ---- Head2EEGMat (assembleSensors.cpp:25-39): nearest triangle by Danielsson's
// point-triangle distance over the interfaces that touch a zero-conductivity
// domain (dist_point_geom, danielsson.cpp:107-128), one CTA per electrode, a
// fixed-order min reduction per interface (candidate segment).  The interfaces
// are visited in the reference's order and each one leaves the weights of its
// own nearest triangle in the shared result, so the electrode's weights are
// those of the last interface's nearest triangle while its triangle is the
// overall nearest (first strictly smaller distance) -- as the reference does.
__global__ void h2em_kernel(const double* __restrict__ pos, int nseg, const int64_t* __restrict__ seg,
                            const int32_t* __restrict__ cand, const double* __restrict__ srec,
                            const int32_t* __restrict__ T, const int64_t* __restrict__ vglob, int64_t nP, int perm,
                            double* dense, int64_t rs, int64_t cs, int64_t col0, int64_t* scols, double* svals) {
    __shared__ double sd[256];
    __shared__ int64_t so[256];
    __shared__ double sa[256][3];
    const int64_t e = blockIdx.x;
    const d3 p = dev::ld3(pos + 3 * e);
    double gbest = 1.79769313486231570e+308, w[3] = {0, 0, 0};
    int64_t gtri = -1;
    for (int q = 0; q < nseg; ++q) {
        double best = 1.79769313486231570e+308, bal[3] = {0, 0, 0};
        int64_t bo = INT64_MAX;
        for (int64_t k = seg[q] + threadIdx.x; k < seg[q + 1]; k += blockDim.x) {
            const double* s = srec + (int64_t)cand[k] * SREC;
            const d3 P[3] = {dev::ld3(s), dev::ld3(s + 3), dev::ld3(s + 6)};
            double al[3];
            const double dist = danielsson_rn(p, P, al);
            if (dist < best) {
                best = dist;
                bo = k;
                bal[0] = al[0]; bal[1] = al[1]; bal[2] = al[2];
            }
        }
        sd[threadIdx.x] = best;
        so[threadIdx.x] = bo;
        sa[threadIdx.x][0] = bal[0]; sa[threadIdx.x][1] = bal[1]; sa[threadIdx.x][2] = bal[2];
        __syncthreads();
        for (int wd = blockDim.x / 2; wd > 0; wd >>= 1) {
            if (threadIdx.x < wd) {
                const int o = threadIdx.x + wd;
                if (sd[o] < sd[threadIdx.x] || (sd[o] == sd[threadIdx.x] && so[o] < so[threadIdx.x])) {
                    sd[threadIdx.x] = sd[o];
                    so[threadIdx.x] = so[o];
                    sa[threadIdx.x][0] = sa[o][0]; sa[threadIdx.x][1] = sa[o][1]; sa[threadIdx.x][2] = sa[o][2];
                }
            }
            __syncthreads();
        }
        if (so[0] != INT64_MAX) {
            if (sd[0] < gbest) {
                gbest = sd[0];
                gtri = cand[so[0]];
            }
            w[0] = sa[0][0]; w[1] = sa[0][1]; w[2] = sa[0][2];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0 && gtri >= 0) {
        for (int j = 0; j < 3; ++j) {
            const int64_t v = vglob ? vglob[T[3 * gtri + j]] : T[3 * gtri + j];   // distinct vertex
            if (dense) dense[(perm ? nP + v : v) * rs + (col0 + e) * cs] = w[j];
            if (scols) scols[3 * e + j] = v;
            if (svals) svals[3 * e + j] = w[j];
        }
    }
}

// ---- Head2MEGMat (assembleSensors.cpp:69-96, assembleFerguson.cpp:18-31,
// operators.h:40-61): OperatorS of every triangle at every sensor, then a
// fixed-order gather per (sensor, vertex) of (B-A) S / (2 A).
__global__ void ferguson_s_kernel(const double* __restrict__ sq, int64_t np, int64_t nt,
                                  const double* __restrict__ srec, double* F) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nt) return;
    for (int64_t i = blockIdx.y; i < np; i += gridDim.y)   // (about 110 FP64 operations; 270 with three atanh and atan2)
        F[i * nt + t] = near_eval<true, false>(srec + t * SREC, dev::ld3(sq + 6 * i), nullptr);
}

__global__ void ferguson_gather_kernel(const double* __restrict__ sq, int64_t np, int64_t nv, int64_t nt,
                                       const double* __restrict__ F, const double* __restrict__ srec,
                                       const int32_t* __restrict__ v2t_beg, const int32_t* __restrict__ v2t_tri,
                                       const int8_t* __restrict__ v2t_loc, const int32_t* __restrict__ tmesh,
                                       const double* __restrict__ jump, int64_t nP, int perm, double* out,
                                       int64_t rs, int64_t cs, int64_t col0, double mag) {
    const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (v >= nv) return;
    for (int64_t i = blockIdx.y; i < np; i += gridDim.y) {
        d3 res = dev::mk(0, 0, 0);
        double coeff = 0.0;
        for (int k = v2t_beg[v]; k < v2t_beg[v + 1]; ++k) {
            const int64_t t = v2t_tri[k];
            const int loc = v2t_loc[k];
            const double* s = srec + t * SREC;
            const d3 A = dev::ld3(s + 3 * ((loc + 1) % 3)), B = dev::ld3(s + 3 * ((loc + 2) % 3));
            res = res + (B - A) * (F[i * nt + t] / (2 * s[12]));
            coeff = jump ? mag * jump[tmesh[t]] : mag;
        }
        const d3 o = dev::ld3(sq + 6 * i + 3);
        out[(perm ? nP + v : v) * rs + (col0 + i) * cs] = dev::dot(res * coeff, o) / dev::norm(o);
    }
}

// ---- DipSource2MEGMat (assembleSensors.cpp:133-159): Biot-Savart primary field.
__global__ void ds2mm_kernel(const double* __restrict__ dip, int64_t nd, const double* __restrict__ sq, int64_t np,
                             double* out, int64_t ldo) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= np) return;
    const d3 o = dev::ld3(sq + 6 * i + 3);
    for (int64_t j = blockIdx.y; j < nd; j += gridDim.y) {
        const d3 r = dev::ld3(dip + 6 * j), q = dev::ld3(dip + 6 * j + 3);
        const d3 diff = dev::ld3(sq + 6 * i) - r;
        const double nd3 = dev::norm(diff);
        const d3 f = dev::cross(q, diff) * (1.0 / (nd3 * nd3 * nd3));
        out[i + j * ldo] = dev::dot(f, o) * kMagFactor / dev::norm(o);
    }
}

void launch_mesh_solid_angles(const double* pts, int64_t pstride, int64_t n, int nmesh, const int64_t* tbeg_dev,
                              const double* srec, double* out, cudaStream_t s, bool screened) {
    if (n == 0) return;
    ProfScope prof_("solid_angles", s);
    if (screened)
        mesh_solid_angles_screened_kernel<<<(unsigned)n, 256, 0, s>>>(pts, pstride, nmesh, tbeg_dev, srec, out);
    else
        mesh_solid_angles_kernel<<<(unsigned)n, 256, 0, s>>>(pts, pstride, nmesh, tbeg_dev, srec, out);
    check_launch("mesh solid angles");
}

void launch_domain_lookup(int64_t n, int nmesh, const double* sa, int ndom, int maxb, const int* dnb,
                          const int* bmesh, const int* binside, const int* borient, const int* bgrp, int forced,
                          int* dom, int* err, cudaStream_t s) {
    ProfScope prof_("domain_lookup", s);
    if (n == 0) return;
    domain_lookup_kernel<<<nblocks(n, 128), 128, 0, s>>>(n, nmesh, sa, ndom, maxb, dnb, bmesh, binside, borient,
                                                         bgrp, forced, dom, err);
    check_launch("domain lookup");
}

// Dipoles whose domain lies outside a planned set (bit d of `allowed`): the
// row ranges of a planned gain contraction would miss their DipSourceMat rows.
// Flags OMG_ERR_INVALID with err[1] = 1 and the first such dipole in err[2].
__global__ void domain_check_kernel(int64_t n, const int* __restrict__ dom, uint64_t allowed, int* err) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int d = dom[i];
    if (d < 0 || (d < 64 && ((allowed >> d) & 1ull))) return;   // d < 0 is flagged by the lookup itself
    if (atomicCAS(err, 0, OMG_ERR_INVALID) == 0) {
        err[1] = 1;
        err[2] = (int)i;
    }
}

void launch_domain_check(int64_t n, const int* dom, uint64_t allowed, int* err, cudaStream_t s) {
    if (n == 0) return;
    domain_check_kernel<<<nblocks(n, 128), 128, 0, s>>>(n, dom, allowed, err);
    check_launch("domain check");
}

static int dsm_sms() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
    }
    return n;
}

void launch_dsm(const DevGeom& g, int64_t dip0, int64_t ndc, const double* dip, const int32_t* tmesh,
                const int64_t* tidx_ref, const int* barrier, const int* orient, const int* dom, int maxb,
                const int* dnb, const int* bmesh, const int* binside, const double* dsigma, int order, int levels,
                double tol, int perm, double* out, int64_t ldo, double* p1tmp, int mixed, cudaStream_t s) {
    ProfScope prof_("dsm", s);
    if (ndc == 0) return;
    if (g.nt >= ((int64_t)1 << DSM_T_BITS) || ndc > INT32_MAX) throw Error(OMG_ERR_UNSUPPORTED, "DSM: too many triangles");
    const bool fp32 = mixed && order == 3 && levels > 0;
    // the pairs the first level does not settle (at most one entry per pair) and their count
    DevBuf left(levels > 0 ? (size_t)ndc * g.nt * sizeof(int2) : 0, s), nleft(sizeof(int), s);
    OMG_CUDA(cudaMemsetAsync(nleft.p, 0, sizeof(int), s));
    const dim3 grid(nblocks(g.nt, 128), (unsigned)ndc);
    if (fp32) {
        DevBuf recf((size_t)g.nt * sizeof(DsmRecF), s);
        dsm_prepare_f_kernel<<<nblocks(g.nt, 128), 128, 0, s>>>(g.nt, g.srec, static_cast<DsmRecF*>(recf.p));
        check_launch("DSM records");
        dsm_mixed_kernel<<<grid, 128, 0, s>>>(dip0, ndc, dip, g.nt, tmesh, tidx_ref, barrier, orient, dom, maxb, dnb, bmesh,
                                              binside, dsigma, tol, g.nvg, perm, out, ldo, p1tmp,
                                              static_cast<const DsmRecF*>(recf.p), left.as<int2>(), nleft.as<int>());
        check_launch("DSM");
    } else {
        constexpr int NPTS[4] = {3, 6, 7, 16};
        const int nsets = levels > 0 ? 5 : 1;
        DevBuf tab((size_t)g.nt * nsets * NPTS[order] * DSM_FL * 8, s);
        DevBuf te((size_t)g.nt * sizeof(int32_t), s);
        dsm_points_kernel<true><<<dim3(nblocks(g.nt, 128), nsets), 128, 0, s>>>(g.nt, g.srec, order, tab.as<double>(),
                                                                                te.as<int32_t>());
        check_launch("DSM points");
        dsm_kernel<<<grid, 128, 0, s>>>(dip0, ndc, dip, g.nt, g.srec, tmesh, tidx_ref, barrier, orient, dom, maxb, dnb, bmesh,
                                        binside, dsigma, order, levels, tol, g.nvg, perm, out, ldo, p1tmp,
                                        tab.as<double>(), te.as<int32_t>(), left.as<int2>(), nleft.as<int>());
        check_launch("DSM");
    }
    if (levels > 0) {
        dsm_fallback_kernel<<<(unsigned)(8 * dsm_sms()), 32 * DSM_WARPS, 0, s>>>(dip0, g.nt, dip, g.srec, tmesh, tidx_ref, orient, dom,
                                                                  maxb, dnb, bmesh, binside, dsigma, order, levels,
                                                                  tol, g.nvg, perm, out, ldo, p1tmp, left.as<int2>(),
                                                                  nleft.as<int>());
        check_launch("DSM (FP64 pairs)");
    }
    dim3 grid2(nblocks(g.nv, 128), (unsigned)ndc);
    dsm_gather_kernel<<<grid2, 128, 0, s>>>(dip0, ndc, g.nv, g.nt, p1tmp, g.v2t_beg, g.v2t_tri, g.v2t_loc, g.nP,
                                            perm, out, ldo);
    check_launch("DSM gather");
}

void launch_h2em(const DevGeom& g, const double* pos, int64_t ne, int nseg, const int64_t* seg, const int32_t* cand,
                 int perm, double* dense, int64_t rs, int64_t cs, int64_t col0, int64_t* scols, double* svals,
                 cudaStream_t s) {
    if (ne == 0) return;
    ProfScope prof_("h2em", s);
    h2em_kernel<<<(unsigned)ne, 256, 0, s>>>(pos, nseg, seg, cand, g.srec, g.T, g.vglob, g.nP, perm, dense, rs, cs,
                                             col0, scols, svals);
    check_launch("H2EM");
}

void launch_h2mm(const DevGeom& g, const double* sq, int64_t np, const int32_t* tmesh, const double* jump, int perm,
                 double* out, int64_t rs, int64_t cs, int64_t col0, double* F, cudaStream_t s, double mag) {
    ProfScope prof_("h2mm", s);
    if (np == 0) return;
    dim3 grid(nblocks(g.nt, 128), (unsigned)std::min<int64_t>(np, 32768));
    ferguson_s_kernel<<<grid, 128, 0, s>>>(sq, np, g.nt, g.srec, F);
    check_launch("Ferguson S");
    dim3 grid2(nblocks(g.nv, 128), (unsigned)std::min<int64_t>(np, 32768));
    ferguson_gather_kernel<<<grid2, 128, 0, s>>>(sq, np, g.nv, g.nt, F, g.srec, g.v2t_beg, g.v2t_tri, g.v2t_loc,
                                                 tmesh, jump, g.nP, perm, out, rs, cs, col0, mag);
    check_launch("Ferguson gather");
}

void launch_ds2mm(const double* dip, int64_t nd, const double* sq, int64_t np, double* out, int64_t ldo,
                  cudaStream_t s) {
    ProfScope prof_("ds2mm", s);
    if (nd == 0 || np == 0) return;
    dim3 grid(nblocks(np, 128), (unsigned)std::min<int64_t>(nd, 32768));
    ds2mm_kernel<<<grid, 128, 0, s>>>(dip, nd, sq, np, out, ldo);
    check_launch("DS2MM");
}

// ===========================================================================
// DipSourceMat vector-Jacobian product: for each dipole j,
//   d/d(r0_j, q_j) of  sum_rows U[row, j] * DSM[row, j]
// from the analytic derivatives of the integrands (Dipole::potential and
// Dipole::gradient, dipole.h:29-46) integrated over the same adaptive trees as
// the forward assembly (integrator.h:228-252): refinement decisions come from
// the forward integrand, so this is the exact derivative of the assembled
// (piecewise) DSM.
// ===========================================================================
struct VjpW {
    double W[3];   // U at the triangle's vertices x coeffD (P1 rows)
    double w0;     // U at the triangle's row x coeffD / sigma (P0 row; 0 on current barriers)
};

// Derivative integrand: kind 0 -> w1(r) * d g / d(r0, q); kind 1 -> w0 * d p / d(r0, q).
__device__ __forceinline__ void dsm_vjp_point(int kind, const DsmTri& T, d3 r0, d3 q, d3 r, const VjpW& w,
                                              double out[6]) {
    const d3 x = r - r0;
    const double inv = 1.0 / dev::dot(x, x);
    const double inv3 = inv * sqrt(inv), inv5 = inv3 * inv, inv7 = inv5 * inv;
    const double qx = dev::dot(q, x);
    if (kind == 1) {
        // p = (q.x)/|x|^3 ; dp/dq = x/|x|^3 ; dp/dr0 = -(q/|x|^3 - 3 (q.x) x/|x|^5)
        const d3 dq = x * inv3;
        const d3 dx = q * inv3 - x * (3.0 * qx * inv5);
        out[0] = -w.w0 * dx.x; out[1] = -w.w0 * dx.y; out[2] = -w.w0 * dx.z;
        out[3] = w.w0 * dq.x; out[4] = w.w0 * dq.y; out[5] = w.w0 * dq.z;
        return;
    }
    const d3 n = T.n;
    const double xn = dev::dot(x, n), qn = dev::dot(q, n);
    // g = (q.n)/|x|^3 - 3 (q.x)(x.n)/|x|^5
    const d3 dq = n * inv3 - x * (3.0 * xn * inv5);
    const d3 dx = x * (-3.0 * qn * inv5 + 15.0 * qx * xn * inv7) - q * (3.0 * xn * inv5) - n * (3.0 * qx * inv5);
    const d3 v = r - T.p0;
    const double a1 = dev::dot(v, T.e10), a2 = dev::dot(v, T.e20);
    const double l1 = T.d11 * a1 + T.d12 * a2, l2 = T.d12 * a1 + T.d22 * a2, l0 = 1.0 - l1 - l2;
    const double w1 = w.W[0] * l0 + w.W[1] * l1 + w.W[2] * l2;
    out[0] = -w1 * dx.x; out[1] = -w1 * dx.y; out[2] = -w1 * dx.z;
    out[3] = w1 * dq.x; out[4] = w1 * dq.y; out[5] = w1 * dq.z;
}

// The weights of a pair.
__device__ __forceinline__ VjpW dsm_vjp_weights(const DsmPair& P, int64_t i, int64_t t, const int32_t* __restrict__ T32,
                                                const int64_t* __restrict__ tidx_ref, const int* __restrict__ barrier,
                                                const double* __restrict__ U, int64_t ldu) {
    const double* Uj = U + i * ldu;
    VjpW w;
    for (int k = 0; k < 3; ++k) w.W[k] = Uj[T32[3 * t + k]] * P.coeffD;
    w.w0 = barrier[P.m] ? 0.0 : Uj[tidx_ref[t]] * (P.coeffD / P.sigma);
    return w;
}

// One thread per (dipole, triangle): the first adaptive level of both
// integrals from the tabled points, as dsm_kernel forms it, and in the same
// pass the derivatives over the points the accepted values sum (54 FP64
// operations per point for both, with one reciprocal square root; the separate
// recursions took ~330); bound by FP64 issue.  100 dipoles on 3840 triangles
// took 1.05 ms after 5.85 with a recursion per pair and integral.  With x = r - r0, y = 1/|x|:
//   g = (q.n) y^3 - 3 (q.x)(n.x) y^5, weighted c1 = w (W0 l0 + W1 l1 + W2 l2):
//     d/dq  = c1 (n y^3 - 3 (n.x) y^5 x),
//     d/dr0 = -c1 ((-3 (q.n) y^5 + 15 (q.x)(n.x) y^7) x - 3 (n.x) y^5 q - 3 (q.x) y^5 n);
//   p = (q.x) y^3, weighted c0 = w w0:
//     d/dq  = c0 y^3 x,   d/dr0 = -c0 (y^3 q - 3 (q.x) y^5 x).
// Pairs not settled are listed as in dsm_kernel; their integral's part is left
// to dsm_vjp_fallback_kernel.
__global__ void dsm_vjp_kernel(int64_t dip0, int64_t ndc, const double* __restrict__ dip, int64_t nt,
                               const double* __restrict__ srec, const int32_t* __restrict__ T32,
                               const int32_t* __restrict__ tmesh, const int64_t* __restrict__ tidx_ref,
                               const int* __restrict__ barrier, const int* __restrict__ orient,
                               const int* __restrict__ dom, int maxb, const int* __restrict__ dnb,
                               const int* __restrict__ bmesh, const int* __restrict__ binside,
                               const double* __restrict__ dsigma, int order, int levels, double tol,
                               const double* __restrict__ U, int64_t ldu, double* part, const double* __restrict__ tab,
                               int2* left, int* nleft) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t il = blockIdx.y;
    if (t >= nt || il >= ndc) return;
    const int64_t i = dip0 + il;
    double* o = part + (il * nt + t) * 6;
    DsmPair P;
    if (!dsm_pair_coeff(i, t, tmesh, orient, dom, maxb, dnb, bmesh, binside, dsigma, P)) {
        for (int c = 0; c < 6; ++c) o[c] = 0.0;
        return;
    }
    const bool p0row = !barrier[P.m];
    const VjpW w = dsm_vjp_weights(P, i, t, T32, tidx_ref, barrier, U, ldu);
    const double* s = srec + t * SREC;
    const d3 n = dev::ld3(s + 9), q = dev::ld3(dip + 6 * i + 3);
    const d3 r0 = dev::ld3(dip + 6 * i), X = r0 * -1.0;   // (added to the tabled points)
    const double h3 = -3.0 * dev::dot(n, (dev::ld3(s) + dev::ld3(s + 3) + dev::ld3(s + 6)) * (1.0 / 3.0) - r0);
    const double qn = dev::dot(q, n), area = s[12], qn3 = -3.0 * qn;
    const double W1 = w.W[1] - w.W[0], W2 = w.W[2] - w.W[0];
    const int np = c_nbpts[order];
    const int64_t set = (int64_t)np * DSM_FL * nt;
    double coarse[4];
    if (levels > 0) dsm_set<false>(tab + t, nt, order, X, q, qn, h3, DsmFix(), coarse);
    double f[4] = {0, 0, 0, 0};                                    // forward sums over the children
    double An = 0, Sq = 0, Sn = 0, Sy = 0;
    d3 Bx = dev::mk(0, 0, 0), Ax = Bx, Cx = Bx, Dx = Bx;
    const double* tb = tab + t + (levels > 0 ? set : 0);
    const int points = (levels > 0 ? 4 : 1) * np;
    for (int j = 0, k = 0; j < points; ++j, k = k + 1 == np ? 0 : k + 1, tb += DSM_FL * nt) {
        const d3 x = dev::mk(X.x + tb[0], X.y + tb[nt], X.z + tb[2 * nt]);
        const double l1 = tb[3 * nt], l2 = tb[4 * nt], t3 = h3 + tb[5 * nt], wk = c_rules[order][k][3];   // t3 = -3 n.x
        const double n2 = fma(x.x, x.x, fma(x.y, x.y, x.z * x.z));
        const double qx = fma(q.x, x.x, fma(q.y, x.y, q.z * x.z));
        double wy;
        const double y = fx::rsqrt64(n2, fx::mant(wk), (int)fx::expo(wk), wk, wy);
        const double y2 = y * y, wy3 = y2 * wy, u = qx * y2, tu = t3 * u;
        const double g = (qn + tu) * wy3;
        f[0] += g;
        f[1] = fma(l1, g, f[1]);
        f[2] = fma(l2, g, f[2]);
        f[3] = fma(qx, wy3, f[3]);
        const double c1 = fma(W1, l1, fma(W2, l2, w.W[0])) * wy3, m = c1 * y2, mt = m * t3;
        An += c1;
        Sq += mt;
        Sn = fma(qx, m, Sn);
        const double ma = m * fma(-5.0, tu, qn3);
        Bx = dev::mk(fma(mt, x.x, Bx.x), fma(mt, x.y, Bx.y), fma(mt, x.z, Bx.z));
        Ax = dev::mk(fma(ma, x.x, Ax.x), fma(ma, x.y, Ax.y), fma(ma, x.z, Ax.z));
        Sy += wy3;
        const double d = wy3 * u;
        Cx = dev::mk(fma(wy3, x.x, Cx.x), fma(wy3, x.y, Cx.y), fma(wy3, x.z, Cx.z));
        Dx = dev::mk(fma(d, x.x, Dx.x), fma(d, x.y, Dx.y), fma(d, x.z, Dx.z));
    }
    bool okv = true, okp = true;
    const double sub = levels > 0 ? 0.25 * area : area;
    if (levels > 0) {   // the test of dsm_kernel
        f[0] -= f[1] + f[2];
        const double lim = dsm_limit(tol);
        double d2 = 0.0, c2 = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const double c = coarse[k] * area, e = c - sub * f[k];
            if (k < 3) {
                d2 = fma(e, e, d2);
                c2 = fma(c, c, c2);
            } else {
                okp = lim >= 0.0 && fabs(e) <= lim * fabs(c);
            }
        }
        okv = lim >= 0.0 && d2 <= lim * lim * c2;
    }
    double g[6] = {0, 0, 0, 0, 0, 0};
    if (okv) {
        const double sn = -3.0 * Sn;
        g[0] = -sub * (Ax.x + q.x * Sq + n.x * sn);
        g[1] = -sub * (Ax.y + q.y * Sq + n.y * sn);
        g[2] = -sub * (Ax.z + q.z * Sq + n.z * sn);
        g[3] = sub * (n.x * An + Bx.x);
        g[4] = sub * (n.y * An + Bx.y);
        g[5] = sub * (n.z * An + Bx.z);
    }
    if (p0row && okp) {
        const double a = sub * w.w0;
        g[0] -= a * (q.x * Sy - 3.0 * Dx.x);
        g[1] -= a * (q.y * Sy - 3.0 * Dx.y);
        g[2] -= a * (q.z * Sy - 3.0 * Dx.z);
        g[3] += a * Cx.x;
        g[4] += a * Cx.y;
        g[5] += a * Cx.z;
    }
    for (int c = 0; c < 6; ++c) o[c] = g[c];
    const int need = (okv ? 0 : 1) | (p0row && !okp ? 2 : 0);
    if (need) left[atomicAdd(nleft, 1)] = make_int2((int)il, (int)t | (need << DSM_T_BITS));
}

// The listed pairs: a warp walks the forward's adaptive tree and adds the
// derivative rule over the children of every accepted node, two points a lane.
__global__ void __launch_bounds__(32 * DSM_WARPS) dsm_vjp_fallback_kernel(
    int64_t dip0, int64_t nt, const double* __restrict__ dip, const double* __restrict__ srec,
    const int32_t* __restrict__ T32, const int32_t* __restrict__ tmesh, const int64_t* __restrict__ tidx_ref,
    const int* __restrict__ barrier, const int* __restrict__ orient, const int* __restrict__ dom, int maxb,
    const int* __restrict__ dnb, const int* __restrict__ bmesh, const int* __restrict__ binside,
    const double* __restrict__ dsigma, int order, int levels, double tol, const double* __restrict__ U, int64_t ldu,
    double* part, const int2* __restrict__ left, const int* __restrict__ nleft) {
    __shared__ DsmNode stack[DSM_WARPS][DSM_STACK];
    const int count = *nleft;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int idx = blockIdx.x * DSM_WARPS + warp; idx < count; idx += gridDim.x * DSM_WARPS) {
        const int2 e = left[idx];
        const int64_t il = e.x, t = e.y & ((1 << DSM_T_BITS) - 1);
        const int need = (int)((unsigned)e.y >> DSM_T_BITS);
        const int64_t i = dip0 + il;
        DsmPair P;
        if (!dsm_pair(i, t, dip, srec, tmesh, orient, dom, maxb, dnb, bmesh, binside, dsigma, P)) continue;
        const VjpW w = dsm_vjp_weights(P, i, t, T32, tidx_ref, barrier, U, ldu);
        double acc[6] = {0, 0, 0, 0, 0, 0};
        for (int kind = 0; kind < 2; ++kind) {
            if (!(need & (1 << kind))) continue;
            dsm_adaptive_warp(kind, order, levels, tol, P.T, P.r0, P.q, P.R0, P.R1, P.R2, P.area, stack[warp], lane,
                              [&](const d3* C, double sub, const double*) {
                                  for (int k = lane & 7; k < c_nbpts[order]; k += 8) {
                                      double d[6];
                                      dsm_vjp_point(kind, P.T, P.r0, P.q, bary_point(c_rules[order][k], C[0], C[1], C[2]),
                                                    w, d);
                                      const double wk = sub * c_rules[order][k][3];
                                      for (int c = 0; c < 6; ++c) acc[c] = fma(wk, d[c], acc[c]);
                                  }
                              });
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            for (int c = 0; c < 6; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
        if (lane == 0)
            for (int c = 0; c < 6; ++c) part[(il * nt + t) * 6 + c] += acc[c];
    }
}

// Fixed-order sum over triangles: one CTA per dipole.
__global__ void dsm_vjp_reduce_kernel(int64_t dip0, int64_t ndc, int64_t nt, const double* __restrict__ part,
                                      double* out) {
    __shared__ double red[6][128];
    const int64_t il = blockIdx.x;
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int64_t t = threadIdx.x; t < nt; t += 128)
        for (int c = 0; c < 6; ++c) acc[c] += part[(il * nt + t) * 6 + c];
    for (int c = 0; c < 6; ++c) red[c][threadIdx.x] = acc[c];
    __syncthreads();
    for (int w = 64; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            for (int c = 0; c < 6; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < 6) out[(dip0 + il) * 6 + threadIdx.x] = red[threadIdx.x][0];
}

void launch_dsm_vjp(const DevGeom& g, int64_t dip0, int64_t ndc, const double* dip, const int32_t* tmesh,
                    const int64_t* tidx_ref, const int* barrier, const int* orient, const int* dom, int maxb,
                    const int* dnb, const int* bmesh, const int* binside, const double* dsigma, int order, int levels,
                    double tol, const double* U, int64_t ldu, double* part, double* out, cudaStream_t s) {
    if (ndc == 0) return;
    ProfScope prof_("dsm_vjp", s);
    if (g.nt >= ((int64_t)1 << DSM_T_BITS) || ndc > INT32_MAX) throw Error(OMG_ERR_UNSUPPORTED, "DSM: too many triangles");
    constexpr int NPTS[4] = {3, 6, 7, 16};
    const int nsets = levels > 0 ? 5 : 1;
    DevBuf tab((size_t)g.nt * nsets * NPTS[order] * DSM_FL * 8, s), nleft(sizeof(int), s),
        left(levels > 0 ? (size_t)ndc * g.nt * sizeof(int2) : 0, s);
    OMG_CUDA(cudaMemsetAsync(nleft.p, 0, sizeof(int), s));
    dsm_points_kernel<false><<<dim3(nblocks(g.nt, 128), nsets), 128, 0, s>>>(g.nt, g.srec, order, tab.as<double>(), nullptr);
    check_launch("DSM points");
    dim3 grid(nblocks(g.nt, 128), (unsigned)ndc);
    dsm_vjp_kernel<<<grid, 128, 0, s>>>(dip0, ndc, dip, g.nt, g.srec, g.T, tmesh, tidx_ref, barrier, orient, dom, maxb,
                                        dnb, bmesh, binside, dsigma, order, levels, tol, U, ldu, part, tab.as<double>(),
                                        left.as<int2>(), nleft.as<int>());
    check_launch("DSM vjp");
    if (levels > 0) {
        dsm_vjp_fallback_kernel<<<(unsigned)(8 * dsm_sms()), 32 * DSM_WARPS, 0, s>>>(
            dip0, g.nt, dip, g.srec, g.T, tmesh, tidx_ref, barrier, orient, dom, maxb, dnb, bmesh, binside, dsigma, order,
            levels, tol, U, ldu, part, left.as<int2>(), nleft.as<int>());
        check_launch("DSM vjp (listed pairs)");
    }
    dsm_vjp_reduce_kernel<<<(unsigned)ndc, 128, 0, s>>>(dip0, ndc, g.nt, part, out);
    check_launch("DSM vjp reduce");
}

// ---------------------------------------------------------------------------
// Internal potentials.  Surf2VolMat (assembleHeadMat.cpp:325-363) through
// PartialBlock (operators.h:302-331): for a point x in a conducting domain and
// every mesh m bounding that domain, with c = K * mesh_orientation(domain, m)
// (domain.h:43-45),
//   row(x), vertex columns   += -c * P1SingleLayerPotential(triangle)(x)[k]
//   row(x), triangle column   =  c / sigma * OperatorS(triangle)(x)   (no current barrier)
// One thread per (triangle, point): the three P1 integrals go to a per-point
// scratch row (zero where the triangle's mesh does not bound the point's
// domain) and the S value straight to its column; a second pass sums the
// scratch over each vertex's triangles in triangle order, as the reference's
// loop accumulates them.  Rows are the kept points (rows[i] >= 0).
// ---------------------------------------------------------------------------
__global__ void partial_block_kernel(int64_t p0, int64_t npc, const double* __restrict__ pts,
                                     const int* __restrict__ pdom, const int64_t* __restrict__ rows, int64_t nt,
                                     const double* __restrict__ srec, const double* __restrict__ prec,
                                     const int32_t* __restrict__ tmesh, const int64_t* __restrict__ tidx_ref,
                                     const int* __restrict__ barrier, const int* __restrict__ orient, int maxb,
                                     const int* __restrict__ dnb, const int* __restrict__ bmesh,
                                     const int* __restrict__ binside, const double* __restrict__ dsigma,
                                     double* __restrict__ p1tmp, double* out, int64_t ldo, int64_t tshift) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t il = blockIdx.y;
    if (t >= nt || il >= npc) return;
    const int64_t i = p0 + il;
    double* o3 = p1tmp + (il * nt + t) * 3;
    o3[0] = o3[1] = o3[2] = 0.0;
    const int64_t row = rows[i];
    if (row < 0) return;
    const int d = pdom[i];
    const int m = tmesh[t];
    double c = 0.0;
    bool on = false;
    for (int k = 0; k < dnb[d]; ++k)
        if (bmesh[d * maxb + k] == m) {
            c = (binside[d * maxb + k] ? kK : -kK) * orient[d * maxb + k];
            on = true;
        }
    if (!on) return;
    const d3 x = dev::ld3(pts + 3 * i);
    double v[3];
    dev::p1_single_layer(prec + t * PREC, x, v);
    o3[0] = v[0] * -c;
    o3[1] = v[1] * -c;
    o3[2] = v[2] * -c;
    if (!barrier[m]) out[row + (tidx_ref[t] + tshift) * ldo] = (c / dsigma[d]) * dev::operator_S(srec + t * SREC, x);
}

__global__ void partial_block_gather_kernel(int64_t p0, int64_t npc, const int64_t* __restrict__ rows, int64_t nv,
                                            int64_t nt, const double* __restrict__ p1tmp,
                                            const int32_t* __restrict__ v2t_beg, const int32_t* __restrict__ v2t_tri,
                                            const int8_t* __restrict__ v2t_loc, double* out, int64_t ldo) {
    const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t il = blockIdx.y;
    if (v >= nv || il >= npc) return;
    const int64_t row = rows[p0 + il];
    if (row < 0) return;
    double sum = 0.0;
    for (int k = v2t_beg[v]; k < v2t_beg[v + 1]; ++k) sum += p1tmp[(il * nt + v2t_tri[k]) * 3 + v2t_loc[k]];
    out[row + v * ldo] = sum;
}

void launch_partial_block(const DevGeom& g, int64_t p0, int64_t npc, const double* pts, const int* pdom,
                          const int64_t* rows, const int32_t* tmesh, const int64_t* tidx_ref, const int* barrier,
                          const int* orient, int maxb, const int* dnb, const int* bmesh, const int* binside,
                          const double* dsigma, double* p1tmp, double* out, int64_t ldo, cudaStream_t s,
                          int64_t tshift) {
    if (npc == 0) return;
    ProfScope prof_("partial_block", s);
    dim3 grid(nblocks(g.nt, 128), (unsigned)npc);
    partial_block_kernel<<<grid, 128, 0, s>>>(p0, npc, pts, pdom, rows, g.nt, g.srec, g.prec, tmesh, tidx_ref,
                                              barrier, orient, maxb, dnb, bmesh, binside, dsigma, p1tmp, out, ldo,
                                              tshift);
    check_launch("partial block");
    dim3 grid2(nblocks(g.nv, 128), (unsigned)npc);
    partial_block_gather_kernel<<<grid2, 128, 0, s>>>(p0, npc, rows, g.nv, g.nt, p1tmp, g.v2t_beg, g.v2t_tri,
                                                      g.v2t_loc, out, ldo);
    check_launch("partial block gather");
}

// DipSource2InternalPotMat (assembleSourceMat.cpp:154-187): the infinite-medium
// potential K / sigma * q.(x - r0) / |x - r0|^3 (dipole.h:29-36) of each
// dipole at each kept point that shares its domain, zero elsewhere.
__global__ void dipole_internal_pot_kernel(const double* __restrict__ pts, const int* __restrict__ pdom,
                                           const int64_t* __restrict__ rows, int64_t np,
                                           const double* __restrict__ dip, const int* __restrict__ ddom, int64_t nd,
                                           const double* __restrict__ dsigma, double* out, int64_t ldo) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= np) return;
    const int64_t row = rows[i];
    if (row < 0) return;
    const int d = pdom[i];
    const d3 x = dev::ld3(pts + 3 * i);
    for (int64_t j = blockIdx.y; j < nd; j += gridDim.y) {
        double val = 0.0;
        if (ddom[j] == d) {
            const d3 r = x - dev::ld3(dip + 6 * j);
            const double n2 = dev::dot(r, r);
            val = (kK / dsigma[d]) * (dev::dot(dev::ld3(dip + 6 * j + 3), r) / (n2 * sqrt(n2)));
        }
        out[row + j * ldo] = val;
    }
}

void launch_dipole_internal_pot(const double* pts, const int* pdom, const int64_t* rows, int64_t np, const double* dip,
                                const int* ddom, int64_t nd, const double* dsigma, double* out, int64_t ldo,
                                cudaStream_t s) {
    if (np == 0 || nd == 0) return;
    ProfScope prof_("dipole_internal_pot", s);
    dim3 grid(nblocks(np, 128), (unsigned)std::min<int64_t>(nd, 32768));
    dipole_internal_pot_kernel<<<grid, 128, 0, s>>>(pts, pdom, rows, np, dip, ddom, nd, dsigma, out, ldo);
    check_launch("dipole internal potential");
}

// ---------------------------------------------------------------------------
// EITSourceMat (assembleSourceMat.cpp:109-152).  The reference fills the
// rows of a transfer matrix for the triangles of current-barrier meshes,
//   D(K o) over (injection triangle, vertices of mesh2)          (operators.h:83-115, 439-442)
//   -1/2 Id on the self pair, Id(t, v) = area / 3                (operators.h:200-206, 267-269)
//   S(-K o sigma_inv) over (injection triangle, triangles of mesh2 != mesh1)   (operators.h:391-425)
// and sums the rows of each electrode's injection triangles with its weight.
// Only the rows of injection triangles are computed here: R is row-major,
// one row of Nref (reference-numbered) columns per injection triangle.
// ---------------------------------------------------------------------------

// Nearest candidate triangle per electrode (dist_point_geom,
// danielsson.cpp:107-128): one CTA per electrode, ties to the first candidate
// (the reference keeps the first strictly smaller distance).
__global__ void nearest_triangle_kernel(const double* __restrict__ pos, int64_t ncand,
                                        const int32_t* __restrict__ cand, const double* __restrict__ srec,
                                        int64_t* out_tri) {
    __shared__ double sd[256];
    __shared__ int64_t so[256];
    const int64_t e = blockIdx.x;
    const d3 p = dev::ld3(pos + 3 * e);
    double best = 1.79769313486231570e+308;
    int64_t bo = INT64_MAX;
    for (int64_t k = threadIdx.x; k < ncand; k += blockDim.x) {
        const double* s = srec + (int64_t)cand[k] * SREC;
        const d3 P[3] = {dev::ld3(s), dev::ld3(s + 3), dev::ld3(s + 6)};
        double al[3];
        const double dist = danielsson_rn(p, P, al);
        if (dist < best) {
            best = dist;
            bo = k;
        }
    }
    sd[threadIdx.x] = best;
    so[threadIdx.x] = bo;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            const int o = threadIdx.x + w;
            if (sd[o] < sd[threadIdx.x] || (sd[o] == sd[threadIdx.x] && so[o] < so[threadIdx.x])) {
                sd[threadIdx.x] = sd[o];
                so[threadIdx.x] = so[o];
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out_tri[e] = so[0] < ncand ? (int64_t)cand[so[0]] : -1;
}

void launch_nearest_triangle(const DevGeom& g, const double* pos, int64_t ne, int64_t ncand, const int32_t* cand,
                             int64_t* out_tri, cudaStream_t s) {
    if (ne == 0) return;
    ProfScope prof_("nearest_triangle", s);
    nearest_triangle_kernel<<<(unsigned)ne, 256, 0, s>>>(pos, ncand, cand, g.srec, out_tri);
    check_launch("nearest triangle");
}

// tmp[(k nb + j) 3 + l] = integral over injection triangle inj[k] of
// P1SingleLayerPotential(t2b + j), component l (the D block's pair integral).
__global__ void eit_d_kernel(const int64_t* __restrict__ inj, int64_t nk, const double* __restrict__ qrec,
                             const double* __restrict__ prec, int64_t t2b, int64_t nb, int order, double* tmp) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t k = blockIdx.y;
    if (j >= nb || k >= nk) return;
    const double* q = qrec + inj[k] * QREC;
    const double* P = prec + (t2b + j) * PREC;
    const int np = c_nbpts[order];
    double acc[3] = {0.0, 0.0, 0.0};
    for (int i = 0; i < np; ++i) {
        double v[3];
        dev::p1_single_layer(P, dev::ld3(q + 3 * i), v);
        const double w = c_rules[order][i][3];
        acc[0] += w * v[0];
        acc[1] += w * v[1];
        acc[2] += w * v[2];
    }
    double* o = tmp + (k * nb + j) * 3;
    o[0] = q[48] * acc[0];
    o[1] = q[48] * acc[1];
    o[2] = q[48] * acc[2];
}

// R[k, v] += coeffD * sum over the triangles of [t2b, t2b + nb) holding v (triangle order),
// then the -1/2 Id term of the self pair.
__global__ void eit_d_gather_kernel(const int64_t* __restrict__ inj, int64_t nk, int64_t t2b, int64_t nb, int64_t vb,
                                    int64_t nvb, double coeffD, int self, const double* __restrict__ tmp,
                                    const int32_t* __restrict__ v2t_beg, const int32_t* __restrict__ v2t_tri,
                                    const int8_t* __restrict__ v2t_loc, const int32_t* __restrict__ T,
                                    const double* __restrict__ srec, const int64_t* __restrict__ vglob, double* R,
                                    int64_t Nref) {
    const int64_t iv = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t k = blockIdx.y;
    if (iv >= nvb || k >= nk) return;
    const int64_t v = vb + iv;
    // the column of the vertex: a copy of a vertex shared by several meshes adds into its distinct vertex
    // (the copies are in different meshes, so different launches, one after the other)
    const int64_t col = vglob ? vglob[v] : v;
    double sum = 0.0;
    for (int q = v2t_beg[v]; q < v2t_beg[v + 1]; ++q) {
        const int64_t t2 = v2t_tri[q];
        if (t2 < t2b || t2 >= t2b + nb) continue;
        sum += tmp[(k * nb + (t2 - t2b)) * 3 + v2t_loc[q]];
    }
    double r = R[k * Nref + col] + coeffD * sum;
    if (self) {
        const int64_t u = inj[k];
        if (T[3 * u] == v || T[3 * u + 1] == v || T[3 * u + 2] == v) r += -0.5 * (srec[u * SREC + 12] / 3.0);
    }
    R[k * Nref + col] = r;
}

// R[k, tidx(t2)] = coeffS * integral over t2 of OperatorS(inj[k]).
__global__ void eit_s_kernel(const int64_t* __restrict__ inj, int64_t nk, const double* __restrict__ srec,
                             const double* __restrict__ qrec, int64_t t2b, int64_t nb, int order,
                             const int64_t* __restrict__ tidx_ref, double coeffS, double* R, int64_t Nref) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t k = blockIdx.y;
    if (j >= nb || k >= nk) return;
    const double* sr = srec + inj[k] * SREC;
    const double* q = qrec + (t2b + j) * QREC;
    const int np = c_nbpts[order];
    double acc = 0.0;
    for (int i = 0; i < np; ++i) acc += c_rules[order][i][3] * dev::operator_S(sr, dev::ld3(q + 3 * i));
    R[k * Nref + tidx_ref[t2b + j]] = (q[48] * acc) * coeffS;
}

void launch_eit_rows(const DevGeom& g, const int64_t* inj, int64_t nk, int64_t t2b, int64_t t2e, int64_t vb,
                     int64_t ve, bool self, bool withS, double coeffD, double coeffS, const int64_t* tidx_ref,
                     int order, double* tmp, double* R, cudaStream_t s) {
    if (nk == 0) return;
    ProfScope prof_("eit_rows", s);
    const int64_t nb = t2e - t2b;
    dim3 grid(nblocks(nb, 128), (unsigned)nk);
    eit_d_kernel<<<grid, 128, 0, s>>>(inj, nk, g.qrec, g.prec, t2b, nb, order, tmp);
    check_launch("EIT D");
    dim3 grid2(nblocks(ve - vb, 128), (unsigned)nk);
    eit_d_gather_kernel<<<grid2, 128, 0, s>>>(inj, nk, t2b, nb, vb, ve - vb, coeffD, self ? 1 : 0, tmp, g.v2t_beg,
                                              g.v2t_tri, g.v2t_loc, g.T, g.srec, g.vglob, R, g.Nref);
    check_launch("EIT D gather");
    if (withS) {
        eit_s_kernel<<<grid, 128, 0, s>>>(inj, nk, g.srec, g.qrec, t2b, nb, order, tidx_ref, coeffS, R, g.Nref);
        check_launch("EIT S");
    }
}

// out[i, e] += sum over the electrode's injection entries q with k0 <= id[q] < k0 + nk
// of coef[q] * R[id[q] - k0, i], in the electrode's triangle order.
__global__ void eit_combine_kernel(int64_t Nref, int64_t ne, const int64_t* __restrict__ ebeg,
                                   const int64_t* __restrict__ eid, const double* __restrict__ ecoef, int64_t k0,
                                   int64_t nk, const double* __restrict__ R, double* out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= Nref) return;
    for (int64_t e = blockIdx.y; e < ne; e += gridDim.y) {
        double acc = out[i + e * Nref];
        for (int64_t q = ebeg[e]; q < ebeg[e + 1]; ++q) {
            const int64_t k = eid[q] - k0;
            if (k >= 0 && k < nk) acc += R[k * Nref + i] * ecoef[q];
        }
        out[i + e * Nref] = acc;
    }
}

void launch_eit_combine(int64_t Nref, int64_t ne, const int64_t* ebeg, const int64_t* eid, const double* ecoef,
                        int64_t k0, int64_t nk, const double* R, double* out, cudaStream_t s) {
    if (ne == 0 || Nref == 0) return;
    ProfScope prof_("eit_combine", s);
    dim3 grid(nblocks(Nref, 256), (unsigned)std::min<int64_t>(ne, 32768));
    eit_combine_kernel<<<grid, 256, 0, s>>>(Nref, ne, ebeg, eid, ecoef, k0, nk, R, out);
    check_launch("EIT combine");
}

// ---------------------------------------------------------------------------
// Shared vertices.  Assembly runs on per-mesh vertex copies (every mesh keeps
// its own vertices, so each block kernel sees a contiguous range); the
// reference's unknowns are the distinct vertices.  With P the copy -> distinct
// vertex map, the reference's head matrix is P^T H P (its N block adds the
// cross-mesh term of a vertex shared by two meshes once with factor 1/2, which
// is the two symmetric copy entries with factor 1/4), its source rows are P^T
// times the copies' rows.  gbeg/gcopy: for distinct vertex u, its copies.
// Internal positions: triangles (and padding) i < nP are their own copies;
// vertex u sits at nP + u (distinct) or nP + v (copy).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void copies_of(int64_t i, int64_t nP, const int64_t* gbeg, const int64_t* gcopy,
                                          int64_t& k0, int64_t& k1) {
    if (i < nP) {
        k0 = -1 - i;   // encodes the single copy i
        k1 = k0 + 1;
    } else {
        k0 = gbeg[i - nP];
        k1 = gbeg[i - nP + 1];
    }
}
__device__ __forceinline__ int64_t copy_at(int64_t k, int64_t nP, const int64_t* gcopy) {
    return k < 0 ? -1 - k : nP + gcopy[k];
}

// Hg (lower triangle, Ng x Ng) = P^T Hl P from the lower triangle of Hl (symmetric).
__global__ void fold_hm_kernel(int64_t Ng, int64_t nP, const int64_t* __restrict__ gbeg,
                               const int64_t* __restrict__ gcopy, const double* __restrict__ hl, int64_t ldl,
                               double* hg, int64_t ldg) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= Ng) return;
    int64_t a0, a1;
    copies_of(i, nP, gbeg, gcopy, a0, a1);
    for (int64_t j = blockIdx.y; j <= i; j += gridDim.y) {
        int64_t b0, b1;
        copies_of(j, nP, gbeg, gcopy, b0, b1);
        double acc = 0.0;
        for (int64_t ka = a0; ka < a1; ++ka) {
            const int64_t a = copy_at(ka, nP, gcopy);
            for (int64_t kb = b0; kb < b1; ++kb) acc += hl[lower_at(a, copy_at(kb, nP, gcopy), ldl)];
        }
        hg[i + j * ldg] = acc;
    }
}

// out (Ng x ncol) = P^T in (Nl x ncol): rows of the copies summed.
__global__ void fold_rows_kernel(int64_t Ng, int64_t nP, const int64_t* __restrict__ gbeg,
                                 const int64_t* __restrict__ gcopy, int64_t ncol, const double* __restrict__ in,
                                 int64_t ldi, double* out, int64_t ldo) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= Ng) return;
    int64_t a0, a1;
    copies_of(i, nP, gbeg, gcopy, a0, a1);
    for (int64_t c = blockIdx.y; c < ncol; c += gridDim.y) {
        double acc = 0.0;
        for (int64_t k = a0; k < a1; ++k) acc += in[copy_at(k, nP, gcopy) + c * ldi];
        out[i + c * ldo] = acc;
    }
}

void launch_fold_hm(int64_t Ng, int64_t nP, const int64_t* gbeg, const int64_t* gcopy, const double* hl, int64_t ldl,
                    double* hg, int64_t ldg, cudaStream_t s) {
    ProfScope prof_("fold", s);
    dim3 grid(nblocks(Ng, 256), (unsigned)std::min<int64_t>(Ng, 32768));
    fold_hm_kernel<<<grid, 256, 0, s>>>(Ng, nP, gbeg, gcopy, hl, ldl, hg, ldg);
    check_launch("fold head matrix");
}

void launch_fold_rows(int64_t Ng, int64_t nP, const int64_t* gbeg, const int64_t* gcopy, int64_t ncol, const double* in,
                      int64_t ldi, double* out, int64_t ldo, cudaStream_t s) {
    if (ncol <= 0) return;
    ProfScope prof_("fold", s);
    dim3 grid(nblocks(Ng, 256), (unsigned)std::min<int64_t>(ncol, 32768));
    fold_rows_kernel<<<grid, 256, 0, s>>>(Ng, nP, gbeg, gcopy, ncol, in, ldi, out, ldo);
    check_launch("fold rows");
}

// out[r * rs + c * cs] (reference numbering r < Nref: distinct vertices, then
// triangle unknowns) = sum over the copies of unknown r of in[copy + c * ldi]
// (internal copy numbering).
__global__ void fold_to_reference_kernel(int64_t Nref, int64_t nvg, int64_t nP, const int64_t* __restrict__ gbeg,
                                         const int64_t* __restrict__ gcopy, int64_t ncol,
                                         const double* __restrict__ in, int64_t ldi, double* out, int64_t rs,
                                         int64_t cs) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= Nref) return;
    const int64_t i = r < nvg ? nP + r : r - nvg;
    int64_t a0, a1;
    copies_of(i, nP, gbeg, gcopy, a0, a1);
    for (int64_t c = blockIdx.y; c < ncol; c += gridDim.y) {
        double acc = 0.0;
        for (int64_t k = a0; k < a1; ++k) acc += in[copy_at(k, nP, gcopy) + c * ldi];
        out[r * rs + c * cs] = acc;
    }
}

// Columns of a per-copy matrix (nrow x (nv + triangles): vertex copies, then the triangle unknowns) folded to
// the reference's columns (distinct vertices, then triangles): out(:, r) = sum of the copies of vertex r, in
// copy order, for r < nvg; the triangle columns moved.
__global__ void fold_columns_kernel(int64_t nrow, int64_t Nref, int64_t nvg, int64_t nv, const int64_t* __restrict__ gbeg,
                                    const int64_t* __restrict__ gcopy, const double* __restrict__ in, int64_t ldi,
                                    double* out, int64_t ldo) {
    for (int64_t r = blockIdx.y; r < Nref; r += gridDim.y)
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nrow;
             i += (int64_t)gridDim.x * blockDim.x) {
            double acc = 0.0;
            if (r < nvg) {
                for (int64_t k = gbeg[r]; k < gbeg[r + 1]; ++k) acc += in[i + gcopy[k] * ldi];
            } else {
                acc = in[i + (r - nvg + nv) * ldi];
            }
            out[i + r * ldo] = acc;
        }
}

void launch_fold_columns(int64_t nrow, int64_t Nref, int64_t nvg, int64_t nv, const int64_t* gbeg,
                         const int64_t* gcopy, const double* in, int64_t ldi, double* out, int64_t ldo,
                         cudaStream_t s) {
    if (nrow <= 0) return;
    ProfScope prof_("fold", s);
    dim3 grid(nblocks(nrow, 256), (unsigned)std::min<int64_t>(Nref, 32768));
    fold_columns_kernel<<<grid, 256, 0, s>>>(nrow, Nref, nvg, nv, gbeg, gcopy, in, ldi, out, ldo);
    check_launch("fold columns");
}

void launch_fold_to_reference(int64_t Nref, int64_t nvg, int64_t nP, const int64_t* gbeg, const int64_t* gcopy,
                              int64_t ncol, const double* in, int64_t ldi, double* out, int64_t rs, int64_t cs,
                              cudaStream_t s) {
    if (ncol <= 0) return;
    ProfScope prof_("fold", s);
    dim3 grid(nblocks(Nref, 256), (unsigned)std::min<int64_t>(ncol, 32768));
    fold_to_reference_kernel<<<grid, 256, 0, s>>>(Nref, nvg, nP, gbeg, gcopy, ncol, in, ldi, out, rs, cs);
    check_launch("fold to reference");
}

}  // namespace omg

// Test hook (not part of the public header): the functions of fixed64.cuh on device arrays; which = 0 sqrt(a),
// 1 2 atanh(b / a) / b, 2 atan2(b, a), with the weight wr where it is not 0; 3 1 / sqrt(a), 4 the weight times it.
namespace omg {
__global__ void fixed64_eval_kernel(int which, int64_t n, const double* a, const double* b, double wr, double* out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t wm = fx::mant(wr);
    const int we = (int)fx::expo(wr);
    if (which == 0)
        out[i] = fx::sqrt64(a[i]);
    else if (which == 1)
        out[i] = wr != 0.0 ? fx::edge<true>(a[i], b[i], wm, we, wr) : fx::edge<false>(a[i], b[i], 0, 0, 0.0);
    else if (which == 2)
        out[i] = wr != 0.0 ? fx::half_angle<true>(b[i], a[i], wm, we, wr) : fx::half_angle<false>(b[i], a[i], 0, 0, 0.0);
    else {
        double wy;
        const double y = fx::rsqrt64(a[i], wm, we, wr, wy);
        out[i] = which == 3 ? y : wy;
    }
}
}  // namespace omg
extern "C" int omg_internal_fixed64(int which, int64_t n, const double* a, const double* b, double wr, double* out) {
    if (n <= 0 || which < 0 || which > 4) return OMG_ERR_INVALID;
    omg::fixed64_eval_kernel<<<omg::nblocks(n, 128), 128>>>(which, n, a, b, wr, out);
    return cudaDeviceSynchronize() == cudaSuccess ? OMG_OK : OMG_ERR_CUDA;
}
