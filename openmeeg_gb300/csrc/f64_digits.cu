// FP64-accurate products on the bf16 tensor cores (sm_103a, tcgen05), for the FP64
// factorization, its solves and general products: the rows of A and B are cut into
// exact fixed-point digits (the scheme of Ozaki, Ogita, Oishi and Rump, Numer.
// Algorithms 59, 2012):
//
//   A_ik = 2^(e_i) sum_{s=1..ND} 2^(-8 s) a_s,ik,  a_s integers, |a_s| <= 128,
//   (A B^T)_ij = 2^(e_i + e_j) sum_l 2^(-8 l) v_l,  v_l = sum_{s+t=l} sum_k a_s,ik b_t,jk.
//
// FP64's own pipe does 1.06 TFLOP/s here, the bf16 tensor cores 1.9 PFLOP/s, so 34
// products are still ~50 times cheaper.
//
// Updates of the factorization and the solves: ND = 7, levels l = 2..9 (34 pairs), an
// entry held to 2^-57 of twice its row's maximum.  |L_i| <= sqrt(a_ii) for the rows of
// a factor, so what is left out is of the size of the factorization's own rounding.
// With l = 9 left out (28 pairs) a solve against a head matrix was three times further
// off than FP64 products.
//
// General products: ND = 8, levels 2..10 (43 pairs), an entry held to 2^-65 of four
// times the maximum of its row's segment of 256.  Rows of potentials and of sources have
// peaks 100 and more above most of their entries, so with seven digits most entries of a
// gain had a larger error bound than K 2^-53 sum |a||b|, FP64's.  With eight the
// errors are below those of FP64 multiply-adds.  For operands graded beyond that, the
// product of the leading digits' magnitudes (one more pair) bounds sum |a||b| from below,
// and an entry whose bound is above FP64's is summed in FP64.
//
// Sums: a product of two digits is at most 2^14, K is at most 256, so the levels up to
// the sixth (general: the eighth) are sums of integers within 2^24, or twice that where
// all digits are as large as they can be, and exact in the FP32 accumulators.  The levels
// 7-9 (9 and 10) share one (the digit planes carry their power of two, so a product
// already has its level's scale): FP32 rounds there by some 2^-56 (2^-72) of the
// exponents' unit in all (measured at K = 256: standard deviation 2^-56.4).
//
// One output tile of 128 x TN is three units of work (general: five), each with two
// accumulators (a half of TMEM's 512 columns, the units alternate between the halves, so
// a unit's products run while the one before is drained): levels {6, 7-9}, {4, 5},
// {2, 3} (general: the magnitudes, {8-10}, {6, 7}, {4, 5}, {2, 3}).
// Within a unit, the K chunks of 64 stream their digit tiles through a ring of 13
// slots of 16 KB, each digit tile of A and of B loaded once per chunk: for s = 1..ND
// the tiles B_t with lmin <= s + t <= lmax slide from high to low t, so at most four B
// tiles and one A tile are live (26 tile loads per chunk and output tile against 68 when
// every pair streams its own).  The epilogue sums an entry from the lowest levels up in
// one 64-bit integer, to 2^-61 (2^-69) of the unit or 2^-60 of the entry, and makes the
// FP64 value by integer operations: the FP64 pipe does one subtraction per entry (at three
// operations it took longer than the products at K = 128).  At 2^-53 of the unit this
// rounding was the largest error of the whole product.
// Output tiles run in super-columns of 12 tile columns, row by row, so the CTAs at
// work at a time share their digit tiles in L2.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "digits.cuh"
#include "fixed64.cuh"
#include "handles.h"
#include "tcgen05.cuh"

namespace omg {

template <typename T>
void negate_rows(T* B, int64_t ldb, int64_t r0, int64_t r1, int64_t n, cudaStream_t s);
template <typename T>
void gemm(int64_t M, int64_t N, int64_t K, T alpha, const T* A, int64_t lda, bool ta, const T* B, int64_t ldb, bool tb,
          T beta, T* C, int64_t ldc, cudaStream_t s, bool lower = false, int64_t row0 = 0, int64_t col0 = 0);

namespace f64d {

using tc::fence_after;
using tc::fence_before;

constexpr int ND7 = 7, ND8 = 8;                   // digits per entry, base 2^8: updates, general products
__host__ __device__ constexpr int planes(int nd) { return nd == ND8 ? 9 : nd; }   // ... and the magnitudes of the first digit
constexpr int BT = 128;                           // tile rows and columns
constexpr int BK = 64;                            // K per chunk: 128-byte swizzled rows
constexpr int SLOT = BT * BK * 2;                 // 16 KB
constexpr int STAGES = 13;
constexpr int EPI_WARPS = 16;
constexpr int THREADS = 64 + EPI_WARPS * 32;      // 576
constexpr int SMEM_BYTES = STAGES * SLOT + 1024;
constexpr uint32_t TMEM_COLS = 512;
constexpr int SUPER = 12;                         // tile columns per super-column
constexpr int EXP_ZERO = -(1 << 20);              // exponent of a zero row: its scale flushes to zero
constexpr int EXP_NAN = 1 << 20;                  // a row with an infinity or a NaN: its outputs become NaN

static inline void check(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw Error(OMG_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
    count_launch();
}

// Programmatic dependent launch (~2 us per launch of a chain): a kernel starts while its predecessor drains and waits for
// it (pdl_wait) before it reads anything that or an earlier kernel wrote; pdl_next lets the successor start before the
// end.  Kernels with several CTAs per SM are launched the ordinary way: launched early, their CTAs crowd onto the SMs that
// are free at that moment (four panel32 + panel_update32 pairs took 296 instead of 150 us at 4400 rows).  What a kernel
// reads after pdl_wait is never __restrict__ const or __ldg: the compiler may move those loads above the wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
static void launch(void (*kern)(KArgs...), dim3 grid, unsigned block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, (KArgs)args...);
}

// Exponent and binary places of a row's digits, from the bits of its largest magnitude: x = 2^e sum_s 2^(-8 s) a_s with
// |x| 2^-e below 1/2 (eight digits: 1/4, so that the integer of 64 places stays below 2^62).
template <int ND>
struct RowScale {
    int e, sh;
    bool finite;
    __device__ __forceinline__ explicit RowScale(unsigned long long mb) {
        const int be = (int)(mb >> 52);
        finite = be < 0x7FF;
        e = mb == 0 ? EXP_ZERO : (finite ? (be ? be : 1) - (ND == ND8 ? 1020 : 1021) : EXP_NAN);
        sh = mb == 0 || !finite ? 0 : 8 * ND - e;
    }
    // the digits of x as one integer: balanced digits without carries by 128 sum_{j < ND - 1} 2^(8 j)
    __device__ __forceinline__ long long digits(double x) const {
        return (finite ? tcr::scaled_rn(x, sh) : 0ll) + (ND == ND8 ? 0x0080808080808080ll : 0x0000808080808080ll);
    }
    // digit s (from 0) of such an integer
    __device__ __forceinline__ static int digit(long long Z, int s) {
        const int bit = 8 * (ND - 1 - s);
        return s == 0 ? (int)(Z >> bit) : (int)((unsigned)(Z >> bit) & 255u) - 128;
    }
};
// 2^(-8 s) d, an FP32 value whose upper half is its bf16
__device__ __forceinline__ unsigned digit_bits(int d, int s) {
    return __float_as_uint((__int_as_float(0x4B400000 + d) - 12582912.0f) * __int_as_float((127 - 8 * s) << 23));
}

// Digits of PER consecutive entries of a row whose largest magnitude has the bits mb, at the entry's place in plane 0
// (planes `plane` entries apart); the row's exponent to *ex.
template <int ND, int PER>
__device__ __forceinline__ void row_digits(const double (&x)[PER], unsigned long long mb, __nv_bfloat16* o, int64_t plane,
                                           int* ex) {
    const RowScale<ND> R(mb);
    if (ex) *ex = R.e;
#pragma unroll
    for (int i0 = 0; i0 < PER; i0 += 8) {
        long long Z[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) Z[u] = R.digits(x[i0 + u]);
#pragma unroll
        for (int s = 0; s < planes(ND); ++s) {   // (plane 8: |a_1|)
            unsigned f[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int d = R.digit(Z[u], s < ND ? s : 0);
                f[u] = digit_bits(s < ND ? d : abs(d), s < ND ? s : 0);
            }
            *reinterpret_cast<uint4*>(o + (int64_t)s * plane + i0) =
                make_uint4(__byte_perm(f[0], f[1], 0x7632), __byte_perm(f[2], f[3], 0x7632),
                           __byte_perm(f[4], f[5], 0x7632), __byte_perm(f[6], f[7], 0x7632));
        }
    }
}

// ---------------------------------------------------------------------------
// Digits of the rows of a column-major m x k matrix in segments of K columns
// (blockIdx.y; 128 or 256, zero-padded): plane s - 1 holds a_s 2^(-8 (s - 1)) in bf16 (exact), rows of `ldk`
// entries; ex[i]: the row's exponent.  A CTA takes 32 rows, lanes along them
// (coalesced reads of the columns), eight groups of K / 8 consecutive columns.
// ---------------------------------------------------------------------------
template <int ND, int K>
__global__ void __launch_bounds__(256) row_digits_kernel(const double* A, int64_t lda, int64_t m, int64_t k,
                                                         int64_t rows_per_plane, __nv_bfloat16* out, int* ex) {
    constexpr int PER = K / 8;
    __shared__ unsigned long long red[8][32];
    const int lane = threadIdx.x % 32, grp = threadIdx.x / 32;
    const int64_t row = (int64_t)blockIdx.x * 32 + lane, c0 = (int64_t)blockIdx.y * K;
    out += (int64_t)blockIdx.y * planes(ND) * rows_per_plane * K;
    ex += (int64_t)blockIdx.y * rows_per_plane;
    double x[PER];
    unsigned long long mb = 0;
    pdl_wait();
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int64_t c = c0 + grp * PER + i;
        x[i] = row < m && c < k ? A[row + c * lda] : 0.0;
        mb = max(mb, (unsigned long long)__double_as_longlong(x[i]) & 0x7FFFFFFFFFFFFFFFull);
    }
    red[grp][lane] = mb;
    __syncthreads();
#pragma unroll
    for (int g = 0; g < 8; ++g) mb = max(mb, red[g][lane]);
    if (row >= m) return;
    row_digits<ND, PER>(x, mb, out + row * K + grp * PER, rows_per_plane * K, grp == 0 ? ex + row : nullptr);
}

// ---------------------------------------------------------------------------
// The product kernel
// ---------------------------------------------------------------------------
// Instruction descriptor: D = F32, A = B = BF16, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BT >> 4) << 24);
}

// The four K = 16 steps of a 64-wide chunk, issued by the lane that holds `lead`.  The whole warp computes the operands: with
// a branch of one lane around each step a step took ~100 cycles.
__device__ __forceinline__ void mma_chunk4(uint32_t tmem, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate, uint32_t lead) {
    asm volatile(
        "{\n .reg .pred p, q, t;\n .reg .b64 a1, a2, a3, b1, b2, b3;\n"
        " setp.ne.b32 q, %5, 0;\n setp.ne.b32 p, %4, 0;\n setp.eq.b32 t, 0, 0;\n"
        " add.u64 a1, %1, 2;\n add.u64 b1, %2, 2;\n add.u64 a2, %1, 4;\n add.u64 b2, %2, 4;\n add.u64 a3, %1, 6;\n add.u64 b3, %2, 6;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, t;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, t;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, t;\n}\n" ::"r"(tmem),
        "l"(a), "l"(b), "r"(id), "r"(accumulate), "r"(lead));
}

__device__ __forceinline__ void commit_by(uint64_t* bar, uint32_t lead) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(dev::smem_u32(bar)),
        "r"(lead)
        : "memory");
}

// T 2^e rounded to nearest even, by integer operations: the FP64 pipe (1/64 of the FP32 rate) is left one subtraction per
// entry.  |T| < 2^63; an exponent past the range of normal numbers flushes to zero or infinity, EXP_NAN gives a NaN.
__device__ __forceinline__ double scaled_double(long long T, int e) {
    if (e > (1 << 19)) return __longlong_as_double(0x7FF8000000000000ll);
    const unsigned long long u = (unsigned long long)(T < 0 ? -T : T);
    const int lz = __clzll((long long)u);
    const unsigned long long m = u << (lz & 63);
    unsigned long long q = m >> 11;   // 53 bits with the leading one
    const unsigned r = (unsigned)m & 0x7FFu;
    q += (r > 0x400u || (r == 0x400u && (q & 1ull))) ? 1ull : 0ull;
    const int ex = e + 1023 + 63 - lz;
    unsigned long long bits = ((unsigned long long)(unsigned)(ex - 1) << 52) + q;   // (a carry moves to the exponent)
    if (u == 0ull || ex <= 0) bits = 0ull;
    else if (ex >= 2047) bits = 0x7FF0000000000000ull;
    return __longlong_as_double((long long)(bits | ((unsigned long long)T & 0x8000000000000000ull)));
}

// The order of a unit's tiles (levels LMIN..LMAX): step s = 1..smax loads the B_t not yet loaded, then A_s, and
// multiplies A_s by B_t for t = tlo(s)..thi(s).
template <int ND, int LMIN, int LMAX>
struct Unit {
    __host__ __device__ static constexpr int least(int a, int b) { return a < b ? a : b; }
    static constexpr int smax = LMAX - 1 < ND ? LMAX - 1 : ND;
    __host__ __device__ static constexpr int tlo(int s) { return LMIN - s > 1 ? LMIN - s : 1; }
    __host__ __device__ static constexpr int thi(int s) { return least(LMAX - s, ND); }
    // the steps that use B_t first and last
    __host__ __device__ static constexpr int first_use(int t) { return t >= tlo(1) ? 1 : LMIN - t; }
    __host__ __device__ static constexpr int last_use(int t) { return least(LMAX - t, smax); }
    // positions of B_t and A_s in the load order
    __host__ __device__ static constexpr int pos_b(int t) { return first_use(t) - 1 + thi(1) - t; }
    __host__ __device__ static constexpr int pos_a(int s) { return s - 1 + thi(1) - tlo(s) + 1; }
    static constexpr int loads = smax + thi(1);
};

struct Ring {
    uint32_t slot, phase, count;   // of the next load; loads issued (producer)
    __device__ __forceinline__ void at(int pos, uint32_t& s, uint32_t& ph) const {
        s = slot + pos;
        ph = phase;
        if (s >= STAGES) {
            s -= STAGES;
            ph ^= 1u;
        }
        if (s >= STAGES) {   // (a unit's loads can pass the end twice)
            s -= STAGES;
            ph ^= 1u;
        }
    }
    __device__ __forceinline__ void advance(int n) {
        uint32_t s, p;
        at(n, s, p);
        slot = s;
        phase = p;
    }
};

struct Shared {
    uint64_t full[STAGES], empty[STAGES], tfull[2], tempty[2], fin;
    uint32_t tmem;
    volatile int abort;
    uint32_t issued;   // loads issued (load g goes to slot g % STAGES), written when the producer ends
};

// The loads of one chunk: unit LMIN..LMAX's digit tiles in their order, or (LMIN = 0) the tiles of plane ND, the magnitudes.
template <int TN, int ND, int LMIN, int LMAX>
__device__ __forceinline__ bool load_chunk(Shared& sh, Ring& r, uint32_t sbase, const CUtensorMap* tA,
                                           const CUtensorMap* tB, int x, int ya, int yb, int ra, int rb) {
    using U = Unit<ND, LMIN, LMAX>;
    auto load = [&](const CUtensorMap* map, int pos, int y, int bytes) -> bool {
        uint32_t s, ph;
        r.at(pos, s, ph);
        if (!tc::wait_or_abort(&sh.empty[s], ph ^ 1u, &sh.abort)) return false;
        dev::mbar_expect_tx(&sh.full[s], bytes);
        tc::tma_load_2d(sbase + s * SLOT, map, x, y, &sh.full[s]);
        ++r.count;
        return true;
    };
    if (LMIN == 0) {
        if (!load(tB, 0, ND * rb + yb, TN * BK * 2) || !load(tA, 1, ND * ra + ya, SLOT)) return false;
        r.advance(2);
        return true;
    }
#pragma unroll
    for (int s = 1; s <= U::smax; ++s) {
#pragma unroll
        for (int t = U::thi(s); t >= U::tlo(s); --t)
            if (U::first_use(t) == s && !load(tB, U::pos_b(t), (t - 1) * rb + yb, TN * BK * 2)) return false;
        if (!load(tA, U::pos_a(s), (s - 1) * ra + ya, SLOT)) return false;
    }
    r.advance(U::loads);
    return true;
}

// The products of one chunk (called by the whole warp); levels LMIN into accumulator 0, the others into accumulator 1.
// FIRST: the unit's first chunk, whose first product of each accumulator overwrites it.
template <int TN, int ND, int LMIN, int LMAX, bool FIRST>
__device__ __forceinline__ bool mma_chunk(Shared& sh, Ring& r, uint32_t sbase, uint32_t acc, uint32_t lead) {
    using U = Unit<ND, LMIN, LMAX>;
    auto wait = [&](int pos, uint32_t& s) -> bool {
        uint32_t ph;
        r.at(pos, s, ph);
        return tc::wait_or_abort(&sh.full[s], ph, &sh.abort);
    };
    if (LMIN == 0) {
        uint32_t sa, sb;
        if (!wait(0, sb) || !wait(1, sa)) return false;
        fence_after();
        mma_chunk4(acc, tc::sdesc_sw128(sbase + sa * SLOT), tc::sdesc_sw128(sbase + sb * SLOT), idesc(TN), FIRST ? 0u : 1u, lead);
        commit_by(&sh.empty[sa], lead);
        commit_by(&sh.empty[sb], lead);
        r.advance(2);
        return true;
    }
    bool fresh0 = FIRST, fresh1 = FIRST;   // resolved at compile time after unrolling
#pragma unroll
    for (int s = 1; s <= U::smax; ++s) {
        uint32_t sa, sb, ph;
#pragma unroll
        for (int t = U::thi(s); t >= U::tlo(s); --t)
            if (U::first_use(t) == s && !wait(U::pos_b(t), sb)) return false;
        if (!wait(U::pos_a(s), sa)) return false;
        fence_after();
        const uint64_t dA = tc::sdesc_sw128(sbase + sa * SLOT);
#pragma unroll
        for (int t = U::thi(s); t >= U::tlo(s); --t) {
            r.at(U::pos_b(t), sb, ph);
            const uint64_t dB = tc::sdesc_sw128(sbase + sb * SLOT);
            const bool hi = s + t == LMIN;
            mma_chunk4(acc + (hi ? 0 : TN), dA, dB, idesc(TN), (hi ? fresh0 : fresh1) ? 0u : 1u, lead);
            if (hi)
                fresh0 = false;
            else
                fresh1 = false;
        }
        commit_by(&sh.empty[sa], lead);
#pragma unroll
        for (int t = U::thi(s); t >= U::tlo(s); --t)
            if (U::last_use(t) == s) {
                r.at(U::pos_b(t), sb, ph);
                commit_by(&sh.empty[sb], lead);
            }
    }
    r.advance(U::loads);
    return true;
}

template <int TN, int ND, int LMIN, int LMAX>
__device__ __forceinline__ bool mma_unit(Shared& sh, Ring& r, uint32_t sbase, uint32_t tmem, uint32_t& lu, int nchunk,
                                         uint32_t lead) {
    const uint32_t half = lu & 1u, acc = tmem + half * 256;
    if (!tc::wait_or_abort(&sh.tempty[half], ((lu >> 1) & 1u) ^ 1u, &sh.abort)) return false;
    fence_after();
    if (!mma_chunk<TN, ND, LMIN, LMAX, true>(sh, r, sbase, acc, lead)) return false;
    for (int c = 1; c < nchunk; ++c)
        if (!mma_chunk<TN, ND, LMIN, LMAX, false>(sh, r, sbase, acc, lead)) return false;
    commit_by(&sh.tfull[half], lead);
    ++lu;
    return true;
}

// Output tile number t of the walk: super-columns of SUPER tile columns, row by row inside.  `lower`: only tiles
// with row >= column.
struct Walk {
    int mt, nt, lower;
    int64_t base = 0;   // first tile number of super-column J
    int J = 0;
    __device__ __forceinline__ int width(int j) const { return min(SUPER, nt - j * SUPER); }
    __device__ __forceinline__ int64_t count(int j) const {
        const int w = width(j);
        if (!lower) return (int64_t)mt * w;
        return (int64_t)(mt - j * SUPER) * w - (int64_t)w * (w - 1) / 2;
    }
    __device__ __forceinline__ void tile(int64_t t, int& i, int& j) {
        while (t >= base + count(J)) {
            base += count(J);
            ++J;
        }
        int64_t o = t - base;
        const int w = width(J);
        if (!lower) {
            i = (int)(o / w);
            j = J * SUPER + (int)(o % w);
            return;
        }
        int r = 0;   // rows J SUPER + r with r + 1 < w tiles
        while (r + 1 < w && o > r) {
            o -= r + 1;
            ++r;
        }
        if (r + 1 >= w) {
            r += (int)(o / w);
            o %= w;
        }
        i = J * SUPER + r;
        j = J * SUPER + (int)o;
    }
};

// UPDATE: C -= A B^T; otherwise segment s of the products, C_s = A_s B_s^T, to the s-th of the M x Nc slices of C, and to the
// s-th slice of `mag` the sum of the products of the first digits' magnitudes over 16, at most 255 (operands: 9 planes per
// segment, exponents per segment; tile numbers run over the segments).
template <int TN, bool UPDATE>
__global__ void __launch_bounds__(THREADS, 1)
    digit_update_kernel(const __grid_constant__ CUtensorMap tA, const __grid_constant__ CUtensorMap tB, int64_t M,
                        int64_t Nc, int nchunk, int ra, int rb, const int* exA,
                        const int* exB, double* C, int64_t ldc, uint8_t* mag, int lower, int64_t ntiles, int* err) {
    constexpr int ND = UPDATE ? ND7 : ND8;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ __align__(8) Shared sh;
    const uint32_t sbase = (dev::smem_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            dev::mbar_init(&sh.full[s], 1);
            dev::mbar_init(&sh.empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            dev::mbar_init(&sh.tfull[a], 1);
            dev::mbar_init(&sh.tempty[a], EPI_WARPS);
        }
        dev::mbar_init(&sh.fin, 1);
        sh.abort = 0;
        sh.issued = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dev::smem_u32(&sh.tmem)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    pdl_wait();
    pdl_next();
    const uint32_t tmem = sh.tmem;
    const int64_t per_seg = UPDATE ? ntiles : ((M + BT - 1) / BT) * ((Nc + TN - 1) / TN);
    const Walk walk0{(int)((M + BT - 1) / BT), (int)((Nc + TN - 1) / TN), lower};
    Walk walk = walk0;

    if (warp == 0) {
        if (lane == 0) {   // ---- TMA producer
            Ring r{0, 0, 0};
            bool ok = true;
            for (int64_t t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
                int i, j;
                const int seg = UPDATE ? 0 : (int)(t / per_seg);
                if (!UPDATE) walk = walk0;
                walk.tile(t - seg * per_seg, i, j);
                const int ya = i * BT + seg * planes(ND) * ra, yb = j * TN + seg * planes(ND) * rb;
                if (!UPDATE) {
                    for (int c = 0; c < nchunk && ok; ++c) ok = load_chunk<TN, ND, 0, 0>(sh, r, sbase, &tA, &tB, c * BK, ya, yb, ra, rb);
                    for (int c = 0; c < nchunk && ok; ++c) ok = load_chunk<TN, ND, 8, 10>(sh, r, sbase, &tA, &tB, c * BK, ya, yb, ra, rb);
                }
                for (int c = 0; c < nchunk && ok; ++c)
                    ok = load_chunk<TN, ND, 6, UPDATE ? 9 : 7>(sh, r, sbase, &tA, &tB, c * BK, ya, yb, ra, rb);
                for (int c = 0; c < nchunk && ok; ++c) ok = load_chunk<TN, ND, 4, 5>(sh, r, sbase, &tA, &tB, c * BK, ya, yb, ra, rb);
                for (int c = 0; c < nchunk && ok; ++c) ok = load_chunk<TN, ND, 2, 3>(sh, r, sbase, &tA, &tB, c * BK, ya, yb, ra, rb);
            }
            sh.issued = r.count;
            if (!ok) sh.abort = 1;
        }
    } else if (warp == 1) {
        // ---- MMA issuer: the warp stays together, one lane issues
        Ring r{0, 0, 0};
        bool ok = true;
        uint32_t lu = 0;
        const uint32_t lead = lane == 0 ? 1u : 0u;
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        for (int64_t t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
            ok = (UPDATE || (mma_unit<TN, ND, 0, 0>(sh, r, sbase, tm, lu, nchunk, lead) &&
                             mma_unit<TN, ND, 8, 10>(sh, r, sbase, tm, lu, nchunk, lead))) &&
                 mma_unit<TN, ND, 6, UPDATE ? 9 : 7>(sh, r, sbase, tm, lu, nchunk, lead) &&
                 mma_unit<TN, ND, 4, 5>(sh, r, sbase, tm, lu, nchunk, lead) &&
                 mma_unit<TN, ND, 2, 3>(sh, r, sbase, tm, lu, nchunk, lead);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) sh.abort = 1;
        commit_by(&sh.fin, lead);
        if (!dev::mbar_wait_bounded(&sh.fin, 0)) sh.abort = 1;
    } else {   // ---- epilogue: warp w owns TMEM lanes 32 (w % 4) .. +31 and columns NCW ((w - 2) / 4) .. + NCW - 1
        constexpr int NCW = TN / 4;
        const int q = warp & 3, c0 = ((warp - 2) >> 2) * NCW;
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        uint32_t lu = 0;
        auto begin = [&]() -> bool {
            bool ok = tc::wait_or_abort(&sh.tfull[lu & 1u], (lu >> 1) & 1u, &sh.abort);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok && lane == 0) sh.abort = 1;
            fence_after();
            return ok;
        };
        auto end = [&]() {
            fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&sh.tempty[lu & 1u]);
            ++lu;
        };
        for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
            int ti, tj;
            const int seg = UPDATE ? 0 : (int)(t / per_seg);
            if (!UPDATE) walk = walk0;
            walk.tile(t - seg * per_seg, ti, tj);
            const int64_t row = (int64_t)ti * BT + q * 32 + lane, col0 = (int64_t)tj * TN + c0;
            // the two accumulators of the unit at hand, eight columns at a time
            auto read = [&](int h, uint32_t (&a)[8], uint32_t (&b)[8]) {
                tc::tmem_ld8(tmem + lanes + (lu & 1u) * 256 + c0 + h * 8, a);
                tc::tmem_ld8(tmem + lanes + (lu & 1u) * 256 + TN + c0 + h * 8, b);
            };
            auto whole = [](uint32_t bits, float scale) { return __float2int_rn(__uint_as_float(bits) * scale); };
            const int64_t j1 = min((int64_t)NCW, Nc - col0), jl = row < M ? (lower ? min(j1, row - col0 + 1) : j1) : 0;
            // low: levels 4 and up in units of 2^-LOW, below 2^61 (seven digits: 2^54) in magnitude
            constexpr int LOW = UPDATE ? 61 : 69;
            long long low[NCW];
            if (!UPDATE) {
                uint8_t* const mr = mag + (int64_t)seg * M * Nc + row + col0 * M;
                if (!begin()) break;
#pragma unroll
                for (int h = 0; h < NCW / 8; ++h) {
                    uint32_t a[8];
                    tc::tmem_ld8(tmem + lanes + (lu & 1u) * 256 + c0 + h * 8, a);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (h * 8 + j < jl) mr[(h * 8 + j) * M] = (uint8_t)min((int)(__uint_as_float(a[j]) * 0.0625f), 255);
                }
                end();
                if (!begin()) break;   // levels 8-10
#pragma unroll
                for (int h = 0; h < NCW / 8; ++h) {
                    uint32_t a[8], b[8];
                    read(h, a, b);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        low[h * 8 + j] = __float2int_rn((__uint_as_float(a[j]) + __uint_as_float(b[j])) * 0x1p53f);
                }
                end();
            }
            if (!begin()) break;   // levels 6 and 7 (7-9)
#pragma unroll
            for (int h = 0; h < NCW / 8; ++h) {
                uint32_t a[8], b[8];
                read(h, a, b);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (UPDATE)
                        low[h * 8 + j] = ((long long)whole(a[j], 0x1p32f) << (LOW - 48)) + whole(b[j], 0x1p45f);
                    else
                        low[h * 8 + j] += ((long long)whole(a[j], 0x1p32f) << (LOW - 48)) + ((long long)whole(b[j], 0x1p40f) << (LOW - 56));
                }
            }
            end();
            if (!begin()) break;   // levels 4 and 5
#pragma unroll
            for (int h = 0; h < NCW / 8; ++h) {
                uint32_t a[8], b[8];
                read(h, a, b);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    low[h * 8 + j] += (((long long)whole(a[j], 0x1p16f) << 8) + whole(b[j], 0x1p24f)) << (LOW - 40);
            }
            end();
            if (!begin()) break;   // levels 2 and 3: G in units of 2^-24, |G| < 2^31; then the value
            const int er = row < M ? exA[row + (int64_t)seg * ra] : EXP_ZERO;
            const int* const eb = exB + (int64_t)seg * rb + col0;
            double* const Cr = C + (int64_t)seg * M * Nc + row + col0 * ldc;
#pragma unroll
            for (int h = 0; h < NCW / 8; ++h) {
                uint32_t a[8], b[8];
                read(h, a, b);
                double c[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) c[j] = UPDATE && h * 8 + j < jl ? Cr[(h * 8 + j) * ldc] : 0.0;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (h * 8 + j < jl) {
                        const int G = (whole(a[j], 1.0f) << 8) + whole(b[j], 0x1p8f);
                        // k places fewer where G 2^(LOW - 24) would not stay below 2^61
                        const int k = max(0, LOW - 24 + 32 - __clz(abs(G)) - 61);
                        const long long T = ((long long)G << (LOW - 24 - k)) + (low[h * 8 + j] >> k);
                        const double v = scaled_double(T, er + eb[h * 8 + j] - LOW + k);
                        Cr[(h * 8 + j) * ldc] = UPDATE ? c[j] - v : v;
                    }
            }
            end();
        }
    }
    __syncthreads();
    if (sh.abort) {
        if (threadIdx.x == 0) {
            atomicExch(err, -8 /* OMG_ERR_TIMEOUT */);
            // copies still in flight land before the shared memory is given up (the last one into each slot)
            for (uint32_t k = 0; k < STAGES && k < sh.issued; ++k) {
                const uint32_t g = sh.issued - 1u - k;
                dev::mbar_wait_bounded(&sh.full[g % STAGES], (g / STAGES) & 1u);
            }
        }
        __syncthreads();
    }
    fence_before();
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

// ---------------------------------------------------------------------------
// Sub-panel of 32 columns: Cholesky of the 32 x 32 diagonal block and P <- P L^-T for the m rows below it, 32 rows per
// CTA.  A warp's FP64 instruction takes its quarter of the SM 64 cycles, however few lanes take part, so both halves are
// laid out for few instructions per warp:
//  * every CTA factors the diagonal block itself (cheaper than a launch that only one SM works on).  Warp 0 runs the
//    serial chain, one FP64 instruction per column (the update of the next column) and the column over its pivot on the
//    integer pipe: a_ik <- a_ik - u_i t_k with u the column as it stands and t = u / a_jj; the other seven warps update
//    the rest of the triangle beside it (packed by columns: one run of entries over all lanes; with three warps the first
//    columns waited for them).  The square roots come last;
//  * four of the warps then solve 8 rows each (4 or 2 where m is small), four lanes per row with every fourth column (8 or
//    16, with every 8th or 16th): the entry solved last goes to
//    the row's lanes by a shuffle and is removed from the later ones with the same t; the results are scaled at the end.
// A 64-column version in two launches took 39 + 28 us for 64 columns, four warps with the reciprocals in FP64 27 us for 32
// (between events), this one 24.
// The factored block goes to Ld (other CTAs still read it in A); place_diagonal_kernel puts the blocks into A at the end.
// ---------------------------------------------------------------------------
constexpr int NBD = 32;
constexpr int PANEL_WARPS = 8;   // 4: solver of N = 6646 19.4 ms, 6: 18.8, 8: 18.5, 12: 18.4

template <int LPR>   // lanes per row
__global__ void __launch_bounds__(32 * PANEL_WARPS) panel32_kernel(const double* A, int64_t lda, int n, int64_t m, double* P, double* Ld,
                                                      int* err, int64_t* err_col, int64_t col_offset) {
    constexpr int NE = NBD * (NBD + 1) / 2;
    __shared__ double U[NE];                     // the triangle, packed by columns
    __shared__ __align__(16) double T[NBD][NBD];   // T[j][i]: t of column j, 0 up to row j
    __shared__ double rs[NBD];
    __shared__ unsigned short ik[NE];
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    auto off = [](int j) { return j * NBD - j * (j - 1) / 2; };
    pdl_wait();
    pdl_next();
    for (int j = warp; j < NBD; j += PANEL_WARPS) {
        const int i = lane;
        if (i >= j) {
            const int e = off(j) + i - j;
            ik[e] = (unsigned short)(i | (j << 8));
            U[e] = i < n && j < n ? A[i + (int64_t)j * lda] : (i == j ? 1.0 : 0.0);   // identity past n
        }
        T[j][i] = 0.0;
    }
    // this CTA's rows, on their way while the block is factored
    const int g = lane % LPR;
    const int64_t row = (int64_t)blockIdx.x * (128 / LPR) + warp * (32 / LPR) + lane / LPR;
    const bool live = warp < 4 && row < m;
    double* p = P + (live ? row : 0) + (int64_t)g * lda;
    double x[NBD / LPR];
#pragma unroll
    for (int i = 0; i < NBD / LPR; ++i) x[i] = live ? p[(int64_t)(LPR * i) * lda] : 0.0;
    __syncthreads();
    int bad = NBD;   // warp 0: the first column with a pivot of the wrong sign
    auto pivot = [&](int j, double v) {   // warp 0: column j is final, v its entry of row j + lane
        const long long bits = __double_as_longlong(__shfl_sync(0xffffffffu, v, 0));
        const bool good = bits > 0 && bits <= 0x7FF0000000000000ll;   // d > 0, off the FP64 pipe
        bad = good ? bad : min(bad, j);
        const double d = __longlong_as_double(good ? bits : 0x3FF0000000000000ll);
        // v / d on the integer pipe (rounded once): the chain of dependent FP64 operations it takes there, three for the
        // reciprocal's correction and the product, is twice as long
        uint32_t ym;
        int ye;
        uint64_t c;
        const bool ok = fx::rcp21(d, ym, ye, c);
        const int ve = (int)fx::expo(v);
        double t = fx::pack<true>(fx::mulh(fx::mul21(fx::mant(v), ym), c) | 1, ve ? ve + ye - 1023 + 2 : 0,
                                  (uint32_t)__double2hiint(v) >> 31);
        t = ve == 0x7FF || !ok ? __longlong_as_double(0x7FF8000000000000ll) : t;
        if (lane > 0 && j + lane < NBD) T[j][j + lane] = t;
    };
    if (warp == 0) pivot(0, U[lane]);
    __syncthreads();
    for (int j = 0; j + 1 < NBD; ++j) {
        const double* t = T[j];
        const double* u = U + off(j) - j;              // u[i]: column j
        const int e1 = off(j + 1), e2 = off(j + 2);    // column j + 1, then the rest
        if (warp == 0) {
            const int r = j + 1 + lane;
            const double v = fma(-u[min(r, NBD - 1)], t[j + 1], U[min(e1 + lane, NE - 1)]);
            if (r < NBD) U[e1 + lane] = v;
            pivot(j + 1, v);
        } else {
#pragma unroll 2
            for (int e = e2 + tid - 32; e < NE; e += 32 * (PANEL_WARPS - 1)) {
                const int q = ik[e];
                U[e] = fma(-u[q & 255], t[q >> 8], U[e]);
            }
        }
        __syncthreads();
    }
    if (warp == 0) {   // rs = 1 / sqrt(d): the approximation times the binomial series 1 + e / 2 + 3 e^2 / 8, e = 1 - d y^2
        const double d0 = U[off(lane)];
        const double d = __double_as_longlong(d0) > 0 ? d0 : 1.0;
        double y;
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
        const double e = fma(-(d * y), y, 1.0);
        rs[lane] = fma(y * e, fma(0.375, e, 0.5), y);
        if (blockIdx.x == 0 && lane == 0 && bad < n && atomicCAS(err, 0, -3 /* OMG_ERR_NOT_DEFINITE */) == 0)
            *err_col = col_offset + bad;
    }
    __syncthreads();
    if (blockIdx.x == 0)
        for (int j = warp; j < NBD; j += PANEL_WARPS) Ld[lane + j * NBD] = lane >= j ? U[off(j) + lane - j] * rs[j] : 0.0;
    if (!__any_sync(0xffffffffu, live)) return;
#pragma unroll
    for (int j = 0; j < NBD; ++j) {
        const double xj = __shfl_sync(0xffffffffu, x[j / LPR], (lane & ~(LPR - 1)) | (j & (LPR - 1)));
#pragma unroll
        for (int i = j / LPR + (j % LPR == LPR - 1 ? 1 : 0); i < NBD / LPR; ++i) x[i] = fma(-xj, T[j][LPR * i + g], x[i]);
    }
    if (!live) return;
#pragma unroll
    for (int i = 0; i < NBD / LPR; ++i) p[(int64_t)(LPR * i) * lda] = x[i] * rs[LPR * i + g];
}

// C (m x nc) -= X Y^T, X the m x 32 sub-panel at the rows of C and Y its first nc rows (C starts at row and column
// 32 (b + 1) of a panel, X at the same row): tiles of 16 rows x 32 columns (4.7 us of FP64 work on an SM; at 32 x 32 the
// short updates left SMs idle and the last wave was longer), the whole K staged at once.
__global__ void __launch_bounds__(128) panel_update32_kernel(int64_t m, int nc, const double* X, double* C,
                                                             int64_t ld) {
    __shared__ double sX[NBD][16], sY[NBD][NBD];   // [k][row]
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const int64_t r0 = (int64_t)blockIdx.x * 16;
    const int c0 = blockIdx.y * 32;
    const int nj = nc - c0 < 32 ? nc - c0 : 32;
    if (r0 + 15 < c0) return;   // above the diagonal
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int k = warp * 8 + u;
        if (lane < 16) sX[k][lane] = r0 + lane < m ? X[r0 + lane + (int64_t)k * ld] : 0.0;
        sY[k][lane] = lane < nj ? X[c0 + lane + (int64_t)k * ld] : 0.0;
    }
    const int r = lane % 16, j0 = warp * 8 + lane / 16 * 4;   // the thread's row and four columns
    const bool live = r0 + r < m;
    double acc[4];
    double* c = C + r0 + r + (int64_t)(c0 + j0) * ld;
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] = live && j0 + u < nj ? c[(int64_t)u * ld] : 0.0;
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < NBD; ++k) {
        const double x = sX[k][r];
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] = fma(-x, sY[k][j0 + u], acc[u]);
    }
    if (!live) return;
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (j0 + u < nj) c[(int64_t)u * ld] = acc[u];
}

// The factored diagonal blocks (32 x 32, one after the other) into the lower triangle of A.  Block b covers the columns
// from 32 b on: the panels start on multiples of 128.
__global__ void place_diagonal_kernel(double* A, int64_t lda, int64_t n, const double* __restrict__ Ld) {
    const int64_t k0 = (int64_t)blockIdx.x * NBD;
    const int i = threadIdx.x % 32;
    for (int j = threadIdx.x / 32; j <= i; j += blockDim.x / 32)
        if (k0 + i < n && k0 + j < n) A[k0 + i + (k0 + j) * lda] = Ld[blockIdx.x * (int64_t)(NBD * NBD) + i + j * NBD];
}

// ---------------------------------------------------------------------------
// FP64 solves by 128-row blocks: the diagonal blocks' inverses, their products with the
// right-hand sides, and the digits of everything the updates between blocks take.
// ---------------------------------------------------------------------------
constexpr int NBS = 128;

// Digits of K = 128 consecutive entries held by a warp (lane: entries 4 lane .. 4 lane + 3), written to row `row` of
// the planes.  mb: the largest magnitude's bits over the row.
__device__ __forceinline__ void write_digits4(const double x[4], unsigned long long mb, __nv_bfloat16* out,
                                              int64_t rows_per_plane, int64_t row, int* ex, int lane) {
    const RowScale<ND7> R(mb);
    if (lane == 0) ex[row] = R.e;
    long long Z[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) Z[u] = R.digits(x[u]);
#pragma unroll
    for (int s = 0; s < ND7; ++s) {
        unsigned f[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) f[u] = digit_bits(R.digit(Z[u], s), s);
        *reinterpret_cast<uint2*>(out + ((int64_t)s * rows_per_plane + row) * NBS + 4 * lane) =
            make_uint2(__byte_perm(f[0], f[1], 0x7632), __byte_perm(f[2], f[3], 0x7632));
    }
}

__device__ __forceinline__ unsigned long long warp_max(unsigned long long mb) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, o));
    return mb;
}

// Block b of an n x n factor starts at row 128 b; rows below it (forward) or columns before it (backward).
__device__ __host__ __forceinline__ int64_t below(int64_t n, int64_t b) { return n > (b + 1) * NBS ? n - (b + 1) * NBS : 0; }

// Digit rows of the panels (columns 128 b .., rows below the diagonal block) of blocks b0 + blockIdx.y: block b's
// planes (7 x below(b) rows of 128) follow those of the blocks before it.
__global__ void __launch_bounds__(256) panel_rows_kernel(const double* __restrict__ A, int64_t lda, int64_t n, int b0,
                                                         __nv_bfloat16* out, int* ex) {
    constexpr int PER = NBS / 8;
    __shared__ unsigned long long red[8][32];
    const int64_t b = b0 + blockIdx.y, m = below(n, b);
    if ((int64_t)blockIdx.x * 32 >= m) return;
    int64_t before = 0;   // rows of the blocks before
    for (int64_t i = b0; i < b; ++i) before += below(n, i);
    const int lane = threadIdx.x % 32, grp = threadIdx.x / 32;
    const int64_t row = (int64_t)blockIdx.x * 32 + lane;
    const double* a = A + (b + 1) * NBS + b * NBS * lda;
    double x[PER];
    unsigned long long mb = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        x[i] = row < m ? a[row + (int64_t)(grp * PER + i) * lda] : 0.0;
        mb = max(mb, (unsigned long long)__double_as_longlong(x[i]) & 0x7FFFFFFFFFFFFFFFull);
    }
    red[grp][lane] = mb;
    __syncthreads();
#pragma unroll
    for (int g = 0; g < 8; ++g) mb = max(mb, red[g][lane]);
    if (row >= m) return;
    row_digits<ND7, PER>(x, mb, out + (7 * before + row) * NBS + grp * PER, m * NBS, grp == 0 ? ex + before + row : nullptr);
}

// Digit rows of the block rows (rows 128 b .. , at most 128 of them, columns before) of blocks b0 + blockIdx.y: a warp per
// column, the K direction contiguous in memory.
__global__ void __launch_bounds__(256) block_cols_kernel(const double* __restrict__ A, int64_t lda, int64_t n, int b0,
                                                         __nv_bfloat16* out, int* ex) {
    const int64_t b = b0 + blockIdx.y, nc = b * NBS;
    const int lane = threadIdx.x % 32;
    const int64_t c = (int64_t)blockIdx.x * 8 + threadIdx.x / 32;
    if (c >= nc) return;
    int64_t before = 0;
    for (int64_t i = b0; i < b; ++i) before += i * NBS;
    const int nk = (int)(n - nc < NBS ? n - nc : NBS);
    const double* a = A + nc + c * lda;
    double x[4];
    unsigned long long mb = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        x[u] = 4 * lane + u < nk ? a[4 * lane + u] : 0.0;
        mb = max(mb, (unsigned long long)__double_as_longlong(x[u]) & 0x7FFFFFFFFFFFFFFFull);
    }
    write_digits4(x, warp_max(mb), out + 7 * before * NBS, nc, c, ex + before, lane);
}

// Inverses of the 128 x 128 lower diagonal blocks (identity past n): CTA (b, g) forms 32 columns by forward substitution,
// lanes along the columns, the rows below the solved one shared by the warps.  Inv: column-major; InvT: its transpose.
__global__ void __launch_bounds__(256) inverse128_kernel(const double* __restrict__ A, int64_t lda, int64_t n, double* Inv,
                                                         double* InvT) {
    extern __shared__ __align__(16) double sm[];   // X (row r, 32 columns), then the rows of L from c0 on
    const int64_t b = blockIdx.x, k0 = b * NBS;
    const int c0 = blockIdx.y * 32, nk = (int)(n - k0 < NBS ? n - k0 : NBS), rows = NBS - c0;
    double* X = sm;
    double* L = sm + NBS * 32;   // L[r * (rows + 1) + l], r, l relative to c0
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const double* a = A + k0 + k0 * lda;
    for (int e = threadIdx.x; e < rows * rows; e += 256) {
        const int r = c0 + e % rows, l = c0 + e / rows;
        L[(r - c0) * (rows + 1) + l - c0] = l > r ? 0.0 : (r < nk ? a[r + (int64_t)l * lda] : (r == l ? 1.0 : 0.0));
    }
    for (int r = warp; r < rows; r += 8) X[r * 32 + lane] = r == lane ? 1.0 : 0.0;
    __syncthreads();
    for (int r = threadIdx.x; r < rows; r += 256) L[r * (rows + 1) + r] = 1.0 / L[r * (rows + 1) + r];
    __syncthreads();
    for (int r = 0; r < rows; ++r) {
        // every warp scales the row itself (the same value), warp r % 8 keeps it
        const double x = X[r * 32 + lane] * L[r * (rows + 1) + r];
        for (int i = r + 1 + ((warp - r - 1) & 7); i < rows; i += 8)
            X[i * 32 + lane] = fma(-L[i * (rows + 1) + r], x, X[i * 32 + lane]);
        __syncthreads();
        if (warp == (r & 7)) X[r * 32 + lane] = x;
    }
    __syncthreads();
    double* o = Inv + b * NBS * NBS;
    double* ot = InvT + b * NBS * NBS;
    for (int e = threadIdx.x; e < NBS * 32; e += 256) {
        const int r = e % NBS, c = e / NBS;   // rows fastest: coalesced columns of Inv
        o[r + (int64_t)(c0 + c) * NBS] = r < c0 ? 0.0 : X[(r - c0) * 32 + c];
    }
    for (int e = threadIdx.x; e < NBS * 32; e += 256) {
        const int c = e % 32, r = e / 32;
        ot[c0 + c + (int64_t)r * NBS] = r < c0 ? 0.0 : X[(r - c0) * 32 + c];
    }
}

// x = M b for the rows of a block (nk <= 128 of them) of one right-hand side per CTA, M lower (Inv) or upper (its
// transpose) and 128 x 128, in place, with the digit row of x^T.  Each row group's dot products are halved between two
// warps, paired so that the four FP64 quarters get the same number of operations (16 (g + 1) and 16 (4 - g)).
__global__ void __launch_bounds__(256) diag_apply_kernel(const double* M, int upper, double* B, int64_t ldb,
                                                         int nk, int64_t nrhs, __nv_bfloat16* out, int* ex) {
    __shared__ double sb[NBS], part[2][NBS];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    double* b = B + (int64_t)blockIdx.x * ldb;
    pdl_wait();
    pdl_next();
    if (threadIdx.x < NBS) sb[threadIdx.x] = threadIdx.x < nk ? b[threadIdx.x] : 0.0;
    const int half = warp >> 2, g = half ? 3 - (warp & 3) : warp & 3;   // rows 32 g + lane
    const int len = upper ? 4 - g : g + 1, r = 32 * g + lane;             // 32 len entries of the row, 16 len per half
    const int l0 = (upper ? 32 * g : 0) + half * 16 * len;
    __syncthreads();
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int l = l0; l < l0 + 16 * len; l += 16)
#pragma unroll
        for (int u = 0; u < 16; ++u) acc[u & 3] = fma(M[r + (l + u) * NBS], sb[l + u], acc[u & 3]);
    part[half][r] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    __syncthreads();
    if (warp != 0) return;
    double v[4];
    unsigned long long mb = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int i = 4 * lane + u;
        v[u] = i < nk ? part[0][i] + part[1][i] : 0.0;
        if (i < nk) b[i] = v[u];
        mb = max(mb, (unsigned long long)__double_as_longlong(v[u]) & 0x7FFFFFFFFFFFFFFFull);
    }
    if (out) write_digits4(v, warp_max(mb), out, nrhs, blockIdx.x, ex, lane);
}

// ---------------------------------------------------------------------------
// General products, K in segments of 256
// ---------------------------------------------------------------------------
constexpr int KS = 256;
constexpr int MAXRANGES = 8;
struct RowRanges {   // the K index runs over rows [beg[q], beg[q] + len[q]) one after the other; n = 0: all rows in order
    int n;
    int64_t beg[MAXRANGES], len[MAXRANGES];
    __device__ __forceinline__ int64_t row(int64_t k) const {
        for (int q = 0; q < n; ++q) {
            if (k < len[q]) return beg[q] + k;
            k -= len[q];
        }
        return k;
    }
};

// Digit rows of the n columns of a column-major matrix, K (kdim of its rows) contiguous in memory: a warp per column and
// segment (blockIdx.y), eight entries per lane.
__global__ void __launch_bounds__(256) col_segments_kernel(const double* __restrict__ A, int64_t lda, int64_t n, int64_t kdim,
                                                           const __grid_constant__ RowRanges rr, __nv_bfloat16* out,
                                                           int* ex) {
    const int lane = threadIdx.x % 32;
    const int64_t c = (int64_t)blockIdx.x * 8 + threadIdx.x / 32, seg = blockIdx.y;
    if (c >= n) return;
    const double* a = A + c * lda;
    double x[8];
    unsigned long long mb = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int64_t k = seg * KS + 8 * lane + u;
        x[u] = k < kdim ? a[rr.row(k)] : 0.0;
        mb = max(mb, (unsigned long long)__double_as_longlong(x[u]) & 0x7FFFFFFFFFFFFFFFull);
    }
    row_digits<ND8, 8>(x, warp_max(mb), out + (seg * planes(ND8) * n + c) * KS + 8 * lane, n * KS,
                       lane == 0 ? ex + seg * n + c : nullptr);
}

// C = alpha sum of the segments' products + beta C, in segment order.
//
// With the exponents' unit u = 2^(e_i + e_j) of a segment, the digits leave out at most K 2^-65.5 u of its product, and FP64
// multiply-adds may be off by K 2^-53 sum |a||b|.  `mag` bounds sum |a||b| from below, in units of 2^-12 u, rounded down:
// where its sum over the segments is less than the sum of the units, the digits' bound is not below FP64's, and the entry
// is left to direct_entries_kernel.  So is one whose row of A or of B^T holds an infinity or a NaN, and one in the range
// of subnormal numbers, which the products flush.  These are listed, and marked in mag's first slice.
__global__ void __launch_bounds__(128) sum_segments_kernel(int64_t M, int64_t N, int nseg, const double* __restrict__ P,
                                                           uint8_t* mag, const int* __restrict__ exA,
                                                           const int* __restrict__ exB, double alpha, double beta, double* C,
                                                           int64_t ldc, int* list, int* count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    for (int64_t j = blockIdx.y; j < N; j += gridDim.y) {
        double v = 0.0;
        bool direct = false;
        int top = 2 * EXP_ZERO;
        for (int g = 0; g < nseg; ++g) {
            const int a = exA[(int64_t)g * M + i], b = exB[(int64_t)g * N + j];
            direct |= a == EXP_NAN || b == EXP_NAN;
            if (a != EXP_ZERO && b != EXP_ZERO) top = max(top, a + b);
        }
        float units = 0.0f, sum = 0.0f;
        for (int g = 0; g < nseg; ++g) {
            const int a = exA[(int64_t)g * M + i], b = exB[(int64_t)g * N + j];
            v += P[((int64_t)g * N + j) * M + i];
            if (a == EXP_ZERO || b == EXP_ZERO) continue;
            const float u = __int_as_float((127 + max(min(a + b - top, 0), -126)) << 23);
            units += u;
            sum += u * (float)mag[((int64_t)g * N + j) * M + i];
        }
        direct |= sum < units || (units > 0.0f && top < -960);
        mag[j * M + i] = direct ? 1 : 0;
        if (direct) {
            list[atomicAdd(count, 1)] = (int)(j * M + i);
            continue;
        }
        double* c = C + i + j * ldc;
        *c = beta == 0.0 ? alpha * v : fma(alpha, v, beta * *c);
    }
}

// The entries of the list in FP64: a CTA each, its threads along K, while they are few (a handful per thousand of a
// potential's rows); past one in 64, tiles of 32 x 32 that have any, which take at most what the FP64 kernel takes for the
// whole product.
struct Operand {   // element (i, k) of op(A): p[i * si + row(k) * sk]
    const double* p;
    int64_t si, sk;
};
__global__ void __launch_bounds__(256) direct_entries_kernel(int64_t M, int64_t N, int64_t kdim, Operand A, Operand B,
                                                             const __grid_constant__ RowRanges rr, int64_t k0, double alpha,
                                                             double beta, double* C, int64_t ldc, const uint8_t* mark,
                                                             const int* list, const int* count) {
    __shared__ double red[8], sa[16][33], sb[16][33];
    const int n = *count, tid = threadIdx.x;
    if (n == 0) return;
    if ((int64_t)n * 64 <= M * N) {
        for (int e = blockIdx.x; e < n; e += gridDim.x) {
            const int64_t i = list[e] % M, j = list[e] / M;
            const double* const a = A.p + i * A.si;
            const double* const b = B.p + j * B.si;
            double part[4] = {};
            for (int64_t k = tid; k < kdim; k += 1024)
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (k + 256 * u < kdim) {
                        const int64_t r = rr.row(k0 + k + 256 * u);
                        part[u] = fma(a[r * A.sk], b[r * B.sk], part[u]);
                    }
            double v = (part[0] + part[1]) + (part[2] + part[3]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (tid % 32 == 0) red[tid / 32] = v;
            __syncthreads();
            if (tid == 0) {
                v = ((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]));
                double* c = C + i + j * ldc;
                *c = beta == 0.0 ? alpha * v : fma(alpha, v, beta * *c);
            }
            __syncthreads();
        }
        return;
    }
    const int64_t mt = (M + 31) / 32, nt = (N + 31) / 32;
    const int ti = tid % 32, tj = tid / 32;   // the thread's row and columns tj + 8 u of a tile
    for (int64_t t = blockIdx.x; t < mt * nt; t += gridDim.x) {
        const int64_t i0 = t % mt * 32, j0 = t / mt * 32;
        bool mine[4], any = false;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            mine[u] = i0 + ti < M && j0 + tj + 8 * u < N && mark[(j0 + tj + 8 * u) * M + i0 + ti];
            any |= mine[u];
        }
        if (!__syncthreads_or(any)) continue;
        double v[4] = {};
        for (int64_t kb = 0; kb < kdim; kb += 16) {
            for (int e = tid; e < 512; e += 256) {   // the faster index along the operand's contiguous direction
                const int ia = A.sk == 1 ? e / 16 : e % 32, ka = A.sk == 1 ? e % 16 : e / 32;
                const int jb = B.sk == 1 ? e / 16 : e % 32, kc = B.sk == 1 ? e % 16 : e / 32;
                sa[ka][ia] = kb + ka < kdim && i0 + ia < M ? A.p[(i0 + ia) * A.si + rr.row(k0 + kb + ka) * A.sk] : 0.0;
                sb[kc][jb] = kb + kc < kdim && j0 + jb < N ? B.p[(j0 + jb) * B.si + rr.row(k0 + kb + kc) * B.sk] : 0.0;
            }
            __syncthreads();
            const int nk = (int)(kdim - kb < 16 ? kdim - kb : 16);
            for (int k = 0; k < nk; ++k)
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = fma(sa[k][ti], sb[k][tj + 8 * u], v[u]);
            __syncthreads();
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (mine[u]) {
                double* c = C + i0 + ti + (j0 + tj + 8 * u) * ldc;
                *c = beta == 0.0 ? alpha * v[u] : fma(alpha, v[u], beta * *c);
            }
    }
}

int64_t sm_count() {
    static int n_sm = 0;
    if (!n_sm) {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        n_sm = n > 0 ? n : 1;
    }
    return n_sm;
}

}  // namespace f64d


// Digit rows of a column-major m x k block (k <= kpad; kpad 128 or 256): 7 planes of rows_per_plane rows of kpad bf16.
void row_digits_f64(const double* A, int64_t lda, int64_t m, int k, int kpad, int64_t rows_per_plane, void* out, int* ex,
                    cudaStream_t s) {
    if (m <= 0) return;
    if ((kpad != 128 && kpad != 256) || k > kpad || rows_per_plane < m) throw Error(OMG_ERR_INVALID, "row digits: bad layout");
    ProfScope prof_("f64_digits", s);
    const unsigned grid = (unsigned)((m + 31) / 32);
    auto kern = kpad == 128 ? f64d::row_digits_kernel<f64d::ND7, 128> : f64d::row_digits_kernel<f64d::ND7, 256>;
    f64d::launch(kern, grid, 256, 0, s, A, lda, m, (int64_t)k, rows_per_plane, static_cast<__nv_bfloat16*>(out), ex);
    f64d::check("FP64 row digits");
}

// nseg > 0: the products of nseg segments, to slices of C and of mag; otherwise the update.
static void digit_product(int64_t M, int64_t Nc, int kpad, const void* A, int64_t ra, int64_t a0, const int* exA,
                          const void* B, int64_t rb, int64_t b0, const int* exB, double* C, int64_t ldc, uint8_t* mag,
                          bool lower, int nseg, int* err, cudaStream_t s, const char* name) {
    if (M <= 0 || Nc <= 0) return;
    const int64_t segs = std::max(1, nseg), np = f64d::planes(nseg > 0 ? f64d::ND8 : f64d::ND7);
    if (kpad % f64d::BK || kpad > 256 || segs * np * std::max(ra, rb) > (1ll << 30))
        throw Error(OMG_ERR_UNSUPPORTED, "digit update: bad sizes");
    ProfScope prof_(name, s);
    static int n_sm = 0;
    if (!n_sm) {
        const int n = (int)f64d::sm_count();
        for (auto k : {f64d::digit_update_kernel<128, true>, f64d::digit_update_kernel<64, true>, f64d::digit_update_kernel<32, true>,
                       f64d::digit_update_kernel<128, false>, f64d::digit_update_kernel<64, false>,
                       f64d::digit_update_kernel<32, false>})
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, f64d::SMEM_BYTES);
        n_sm = n;
    }
    // Tile width: narrow tiles put a short product (a solve's right-hand sides, the next panel) on more SMs and leave a
    // shorter last epilogue, wide ones feed the tensor cores better.  Cycles of a tile's products (a K = 16 step takes
    // 64 / 48 / 40 cycles at 128 / 64 / 32 columns: shared memory feeds 128 bytes a cycle) by the number of waves, plus
    // one epilogue of ~100 cycles a column.
    const int64_t mt = (M + f64d::BT - 1) / f64d::BT;
    int tn = 128;
    if (!lower) {
        int64_t best = INT64_MAX;
        for (int w : {128, 64, 32}) {
            const int64_t waves = (segs * mt * ((Nc + w - 1) / w) + n_sm - 1) / n_sm;
            const int64_t t = waves * (nseg > 0 ? 44 : 34) * (kpad / 16) * (w == 128 ? 64 : w == 64 ? 48 : 40) + 100 * w;
            if (t < best) {
                best = t;
                tn = w;
            }
        }
    }
    const CUtensorMap mA = tc::make_map_2d(static_cast<const uint16_t*>(A) + a0 * kpad, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                                           2, segs * np * ra - a0, kpad, kpad, f64d::BK, f64d::BT);
    const CUtensorMap mB = tc::make_map_2d(static_cast<const uint16_t*>(B) + b0 * kpad, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                                           2, segs * np * rb - b0, kpad, kpad, f64d::BK, tn);
    const int64_t nt = (Nc + tn - 1) / tn;
    const int64_t ntiles = segs * (lower ? mt * nt - nt * (nt - 1) / 2 : mt * nt);
    const unsigned grid = (unsigned)std::min<int64_t>(ntiles, n_sm);
    auto kern = nseg > 0 ? (tn == 128  ? f64d::digit_update_kernel<128, false>
                            : tn == 64 ? f64d::digit_update_kernel<64, false>
                                       : f64d::digit_update_kernel<32, false>)
                         : (tn == 128  ? f64d::digit_update_kernel<128, true>
                            : tn == 64 ? f64d::digit_update_kernel<64, true>
                                       : f64d::digit_update_kernel<32, true>);
    f64d::launch(kern, grid, f64d::THREADS, f64d::SMEM_BYTES, s, mA, mB, M, Nc, kpad / f64d::BK, (int)ra, (int)rb, exA + a0,
                 exB + b0, C, ldc, mag, lower ? 1 : 0, ntiles, err);
    f64d::check(name);
}

// C (M x Nc, column-major; `lower`: entries with row >= column only) -= A B^T from digit rows of kpad entries:
// A's planes start at row a0 of buffers of ra rows per plane, B's at b0 of rb.
void digit_update_f64(int64_t M, int64_t Nc, int kpad, const void* A, int64_t ra, int64_t a0, const int* exA,
                      const void* B, int64_t rb, int64_t b0, const int* exB, double* C, int64_t ldc, bool lower,
                      int* err, cudaStream_t s, const char* name) {
    digit_product(M, Nc, kpad, A, ra, a0, exA, B, rb, b0, exB, C, ldc, nullptr, lower, 0, err, s, name);
}

// Whether a general product goes by digit products: where they take less time than the FP64 kernel.  Measured in calls,
// their fixed 16 us taken off: the FP64 kernel 0.29 us per K and wave of 32 x 32 tiles, 1.07 per K for an output within one
// (a 64 x 64 tile on one SM); the digits 88 us (launches, the least product) and per segment of 256 29 us for a million
// entries of C and 17 for a million entries of A and B.  E.g. 64 x 100 x 207: 59 us by FP64, 88 by digits; 64 x 100 x 600 176
// and 88; 1 x 1 x 100 107 and 84; 4486 x 151 x 4486 9459 and 810.
bool gemm_f64_by_digits(int64_t M, int64_t N, int64_t K) {
    if (M <= 0 || N <= 0 || K <= 0) return false;
    const double waves = std::ceil((double)((M + 31) / 32) * (double)((N + 31) / 32) / (double)f64d::sm_count());
    const double fp64_us = (M <= 32 && N <= 32 ? 1.07 : 0.29 * waves) * (double)K;
    const double nseg = (double)((K + f64d::KS - 1) / f64d::KS);
    return fp64_us > 88.0 + nseg * (29e-6 * (double)M * (double)N + 17e-6 * (double)(M + N) * f64d::KS);
}

// C (M x N) = alpha op(A) op(B) + beta C over the K rows (columns) the ranges list (null: all K), FP64, column-major, with an
// error of at most K 2^-53 sum |a||b| per entry.
void gemm_f64(int64_t M, int64_t N, int64_t K, double alpha, const double* A, int64_t lda, bool ta, const double* B,
              int64_t ldb, bool tb, double beta, double* C, int64_t ldc, int* err, cudaStream_t s,
              const std::vector<std::pair<int64_t, int64_t>>* ranges) {
    using namespace f64d;
    if (M <= 0 || N <= 0) return;
    if (ranges && ranges->size() > (size_t)MAXRANGES) {   // (a kernel parameter lists MAXRANGES of them)
        for (size_t q = 0; q < ranges->size(); q += MAXRANGES) {
            const std::vector<std::pair<int64_t, int64_t>> part(ranges->begin() + q,
                                                                ranges->begin() + std::min(q + MAXRANGES, ranges->size()));
            gemm_f64(M, N, 0, alpha, A, lda, ta, B, ldb, tb, q == 0 ? beta : 1.0, C, ldc, err, s, &part);
        }
        return;
    }
    RowRanges rr{};
    if (ranges) {
        K = 0;
        for (const auto& r : *ranges) {
            rr.beg[rr.n] = r.first;
            rr.len[rr.n] = r.second - r.first;
            K += rr.len[rr.n++];
        }
        if (rr.n > 0 && (!ta || tb)) throw Error(OMG_ERR_INVALID, "GEMM: row ranges need both operands K-contiguous");
    }
    if (!gemm_f64_by_digits(M, N, K)) {
        if (K <= 0 || rr.n == 0) {
            gemm<double>(M, N, K, alpha, A, lda, ta, B, ldb, tb, beta, C, ldc, s);
            return;
        }
        for (int q = 0; q < rr.n; ++q)
            gemm<double>(M, N, rr.len[q], alpha, A + rr.beg[q], lda, true, B + rr.beg[q], ldb, false, q == 0 ? beta : 1.0, C,
                         ldc, s);
        return;
    }
    // Blocks of rows and columns, and segments at a time, for which the partial products with their bounds and each
    // operand's digits take 512 MB at most.
    constexpr int64_t MOST = 512ll << 20, DIGIT_ROW = (int64_t)planes(ND8) * KS * 2;
    const int64_t nseg = (K + KS - 1) / KS;
    const int64_t mb = std::min(M, MOST / DIGIT_ROW / BT * BT);
    const int64_t nb = std::min({N, MOST / DIGIT_ROW / BT * BT, std::max<int64_t>(BT, MOST / (mb * 9) / BT * BT)});
    const int64_t at_once = std::max<int64_t>(1, std::min<int64_t>({nseg, 65535, MOST / (mb * nb * 9), MOST / (std::max(mb, nb) * DIGIT_ROW)}));
    DevBuf P((size_t)at_once * mb * nb * 8, s), W((size_t)at_once * mb * nb, s), dA((size_t)at_once * mb * DIGIT_ROW, s),
        dB((size_t)at_once * nb * DIGIT_ROW, s), left((size_t)(mb * nb + 1) * sizeof(int), s), ex((size_t)at_once * (mb + nb) * sizeof(int), s);
    auto block = [&](int64_t M, int64_t N, const double* A, const double* B, double* C) {
        int* exA = ex.as<int>();
        int* exB = exA + at_once * M;
        for (int64_t g0 = 0; g0 < nseg; g0 += at_once) {
            const int64_t ns = std::min(at_once, nseg - g0), k0 = g0 * KS, kk = std::min(K - k0, ns * KS);
            RowRanges part = rr;   // the rows from k0 on
            for (int64_t skip = k0; part.n > 0 && skip > 0;) {
                const int64_t d = std::min(skip, part.len[0]);
                part.beg[0] += d;
                part.len[0] -= d;
                skip -= d;
                if (part.len[0] == 0 && part.n > 1) {
                    for (int q = 1; q < part.n; ++q) {
                        part.beg[q - 1] = part.beg[q];
                        part.len[q - 1] = part.len[q];
                    }
                    --part.n;
                }
            }
            auto digits = [&](const double* X, int64_t ldx, bool k_contiguous, int64_t n, void* out, int* e) {
                ProfScope prof_("f64_digits", s);
                if (k_contiguous)
                    col_segments_kernel<<<dim3((unsigned)((n + 7) / 8), (unsigned)ns), 256, 0, s>>>(
                        X + (part.n ? 0 : k0), ldx, n, kk, part, static_cast<__nv_bfloat16*>(out), e);
                else
                    launch(row_digits_kernel<ND8, KS>, dim3((unsigned)((n + 31) / 32), (unsigned)ns), 256, 0, s, X + k0 * ldx,
                           ldx, n, kk, n, static_cast<__nv_bfloat16*>(out), e);
                check("GEMM digits");
            };
            digits(A, lda, ta, M, dA.p, exA);
            digits(B, ldb, !tb, N, dB.p, exB);
            digit_product(M, N, KS, dA.p, M, 0, exA, dB.p, N, 0, exB, P.as<double>(), M, W.as<uint8_t>(), false, (int)ns, err,
                          s, "f64_product");
            ProfScope prof_("f64_segments", s);
            OMG_CUDA(cudaMemsetAsync(left.p, 0, sizeof(int), s));
            int* count = left.as<int>();
            sum_segments_kernel<<<dim3((unsigned)((M + 127) / 128), (unsigned)std::min<int64_t>(N, 65535)), 128, 0, s>>>(
                M, N, (int)ns, P.as<double>(), W.as<uint8_t>(), exA, exB, alpha, g0 == 0 ? beta : 1.0, C, ldc, count + 1,
                count);
            check("GEMM segments");
            const Operand oa{A, ta ? lda : 1, ta ? 1 : lda}, ob{B, tb ? 1 : ldb, tb ? ldb : 1};
            direct_entries_kernel<<<(unsigned)std::min<int64_t>((M * N + 63) / 64, 4 * sm_count()), 256, 0, s>>>(
                M, N, kk, oa, ob, rr, k0, alpha, g0 == 0 ? beta : 1.0, C, ldc, W.as<uint8_t>(), count + 1, count);
            check("GEMM entries");
        }
    };
    for (int64_t i0 = 0; i0 < M; i0 += mb)
        for (int64_t j0 = 0; j0 < N; j0 += nb)
            block(std::min(mb, M - i0), std::min(nb, N - j0), A + i0 * (ta ? lda : 1), B + j0 * (tb ? 1 : ldb), C + i0 + j0 * ldc);
}

// Sub-panel at (k0, k0) of the matrix, w <= 32 columns: the diagonal block's factor to Ld, the rows below solved in place.
void panel32(double* A, int64_t lda, int w, int64_t m, double* Ld, int* err, int64_t* err_col, int64_t col_offset,
             cudaStream_t s) {
    ProfScope prof_("f64_panel", s);
    // Few rows: more lanes per row, fewer rows per CTA, while one CTA per SM holds them all (the rows' substitution takes a
    // quarter of the SM 144 / 80 / 48 FP64 instructions at 4 / 8 / 16 lanes per row: the smallest gain's 36 sub-panels 0.85 ->
    // 0.71 ms).  With more rows than that, CTAs that share an SM would repeat the triangle.
    const int64_t sms = f64d::sm_count();
    const int lpr = m <= 8 * sms ? 16 : m <= 16 * sms ? 8 : 4;
    auto kern = lpr == 16 ? f64d::panel32_kernel<16> : lpr == 8 ? f64d::panel32_kernel<8> : f64d::panel32_kernel<4>;
    const int64_t rows = 128 / lpr;
    f64d::launch(kern, dim3((unsigned)std::max<int64_t>(1, (m + rows - 1) / rows)), 32 * f64d::PANEL_WARPS, 0, s,
                 (const double*)A, lda, w, m, A + w, Ld, err, err_col, col_offset);
    f64d::check("FP64 panel");
}

// C (m x nc, its first nc rows lower) -= X (m x 32) (first nc rows of X)^T.
void panel_update32(int64_t m, int nc, const double* X, double* C, int64_t ld, cudaStream_t s) {
    if (m <= 0 || nc <= 0) return;
    ProfScope prof_("f64_panel_update", s);
    f64d::panel_update32_kernel<<<dim3((unsigned)((m + 15) / 16), (unsigned)((nc + 31) / 32)), 128, 0, s>>>(m, nc, X, C, ld);
    f64d::check("FP64 panel update");
}

void place_diagonal_f64(double* A, int64_t lda, int64_t n, const double* Ld, cudaStream_t s) {
    if (n <= 0) return;
    f64d::place_diagonal_kernel<<<(unsigned)((n + 31) / 32), 256, 0, s>>>(A, lda, n, Ld);
    f64d::check("FP64 diagonal blocks");
}

// B (n x nrhs) <- (L D L^T)^-1 B with the FP64 factor's lower triangle L (128-row blocks) and D = diag(+I, -I) from row
// nP on; Inv / InvT: the diagonal blocks' inverses (inverse_blocks_f64).  Each sweep is, per block, the product with the
// inverse (FP64 pipe) and one FP64-accurate digit update of all rows still to come.  The factor's digits are formed per
// call, for as many blocks at a time as 2 GB hold.
void solve_f64(int64_t n, int64_t nP, const double* L, int64_t ld, const double* Inv, const double* InvT, double* B,
               int64_t ldb, int64_t nrhs, int* err, cudaStream_t s) {
    using namespace f64d;
    if (n <= 0 || nrhs <= 0) return;
    const int64_t nb = (n + NBS - 1) / NBS;
    auto rows_of = [&](bool fwd, int64_t b) { return fwd ? below(n, b) : b * NBS; };
    const int64_t budget = std::max<int64_t>(2ll << 30, 7 * n * NBS * 2);
    DevBuf xd((size_t)7 * nrhs * NBS * 2, s), xe((size_t)nrhs * sizeof(int), s);
    for (int back = 0; back < 2; ++back) {
        const bool fwd = !back;
        if (back) negate_rows<double>(B, ldb, nP, n, nrhs, s);
        for (int64_t q0 = 0; q0 < nb;) {   // q: position in the sweep
            int64_t q1 = q0, rows = 0;
            auto block = [&](int64_t q) { return fwd ? q : nb - 1 - q; };
            while (q1 < nb && (rows + rows_of(fwd, block(q1))) * 7 * NBS * 2 <= budget) rows += rows_of(fwd, block(q1++));
            const int64_t lo = std::min(block(q0), block(q1 - 1)), cnt = q1 - q0;
            DevBuf dig((size_t)7 * rows * NBS * 2, s), ex((size_t)rows * sizeof(int), s);
            if (rows > 0) {
                ProfScope prof_("f64_digits", s);
                if (fwd)
                    panel_rows_kernel<<<dim3((unsigned)((below(n, lo) + 31) / 32), (unsigned)cnt), 256, 0, s>>>(
                        L, ld, n, (int)lo, dig.as<__nv_bfloat16>(), ex.as<int>());
                else
                    block_cols_kernel<<<dim3((unsigned)(((lo + cnt - 1) * NBS + 7) / 8), (unsigned)cnt), 256, 0, s>>>(
                        L, ld, n, (int)lo, dig.as<__nv_bfloat16>(), ex.as<int>());
                check("factor digits");
            }
            for (int64_t q = q0; q < q1; ++q) {
                const int64_t b = block(q), k0 = b * NBS, m = rows_of(fwd, b);
                const int nk = (int)std::min<int64_t>(NBS, n - k0);
                {
                    ProfScope prof_("f64_diag", s);
                    launch(diag_apply_kernel, dim3((unsigned)nrhs), 256, 0, s, (fwd ? Inv : InvT) + b * NBS * NBS, back,
                           B + k0, ldb, nk, nrhs, m > 0 ? xd.as<__nv_bfloat16>() : nullptr, xe.as<int>());
                    check("diagonal block");
                }
                if (m == 0) continue;
                int64_t before = 0;
                for (int64_t i = lo; i < b; ++i) before += rows_of(fwd, i);
                digit_update_f64(m, nrhs, NBS, dig.as<uint16_t>() + 7 * before * NBS, m, 0, ex.as<int>() + before, xd.p,
                                 nrhs, 0, xe.as<int>(), fwd ? B + k0 + NBS : B, ldb, false, err, s, "f64_solve");
            }
            q0 = q1;
        }
    }
}

// Inverses (and their transposes) of the 128 x 128 diagonal blocks of a lower factor, identity past n.
void inverse_blocks_f64(int64_t n, const double* L, int64_t ld, double* Inv, double* InvT, cudaStream_t s) {
    ProfScope prof_("f64_inverse", s);
    constexpr int SM = (f64d::NBS * 32 + f64d::NBS * (f64d::NBS + 1)) * 8;
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(f64d::inverse128_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SM);
        attr = true;
    }
    f64d::inverse128_kernel<<<dim3((unsigned)((n + f64d::NBS - 1) / f64d::NBS), 4), 256, SM, s>>>(L, ld, n, Inv, InvT);
    f64d::check("diagonal inverses");
}

}  // namespace omg

// Test hook (not part of the public header): C -= A B^T through the digits and the tensor-core kernel; A M x k, B Nc x k,
// C M x Nc (column-major FP64 device pointers, leading dimensions M, Nc, M), k <= 256.
extern "C" int omg_internal_digit_update(int64_t M, int64_t Nc, int k, const double* A, const double* B, double* C,
                                         int lower, int* err) {
    try {
        const int kpad = k <= 128 ? 128 : 256;
        cudaStream_t s = 0;
        DevBuf da((size_t)7 * M * kpad * 2, s), db((size_t)7 * Nc * kpad * 2, s), ea((size_t)M * 4, s), eb((size_t)Nc * 4, s);
        omg::row_digits_f64(A, M, M, k, kpad, M, da.p, ea.as<int>(), s);
        omg::row_digits_f64(B, Nc, Nc, k, kpad, Nc, db.p, eb.as<int>(), s);
        omg::digit_update_f64(M, Nc, kpad, da.p, M, 0, ea.as<int>(), db.p, Nc, 0, eb.as<int>(), C, M, lower != 0, err, s,
                              "digit_update");
        return cudaDeviceSynchronize() == cudaSuccess ? 0 : -2;
    } catch (const omg::Error& e) {
        return e.code;
    }
}

// Test hook: Cholesky of the w x w (w <= 32) block at the top of the (w + m) x w matrix A (column-major) and the rows below
// it <- rows L^-T, in place.
extern "C" int omg_internal_panel32(int w, int64_t m, double* A, int* err, int64_t* err_col) {
    try {
        cudaStream_t s = 0;
        DevBuf Ld(32 * 32 * 8, s);
        omg::panel32(A, w + m, w, m, Ld.as<double>(), err, err_col, 0, s);
        omg::place_diagonal_f64(A, w + m, w, Ld.as<double>(), s);
        return cudaDeviceSynchronize() == cudaSuccess ? 0 : -2;
    } catch (const omg::Error& e) {
        return e.code;
    }
}
