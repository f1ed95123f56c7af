// Square roots, logarithms of edges and solid angles of FP64 values on the
// integer pipe.
//
// A GB300 SM retires 1.7 FP64 results per clock but issues four warp
// instructions: a DFMA holds a warp's quarter of the SM for 76 clocks (a
// conversion or a comparison likewise), in which about 15 IMAD.WIDE issue
// beside it at no cost (measured: four 64-bit high products, 20 clocks each,
// between two DFMAs take the time of the DFMAs).  So whatever follows from a
// hardware approximation by small corrections is computed here in 64-bit fixed
// point: the mantissas are multiplied as integers, the residual of the
// approximation is exact modulo 2^64, and polynomials of a bounded argument
// run in Q64, whose absolute error (2^-60 and less) is below that of FP64.
// The result is rounded once, to nearest.
#pragma once
#include <cstdint>

namespace omg {
namespace fx {

__device__ __forceinline__ uint32_t expo(double x) { return ((uint32_t)__double2hiint(x) >> 20) & 0x7FF; }
// The mantissa with its leading one at bit 63 (normal x).
__device__ __forceinline__ uint64_t mant(double x) {
    return ((uint64_t)__double_as_longlong(x) << 11) | 0x8000000000000000ull;
}
__device__ __forceinline__ uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
__device__ __forceinline__ uint32_t lo32(uint64_t x) { return (uint32_t)x; }

// a b / 2^64 to 2 units (the low product is left out).
__device__ __forceinline__ uint64_t mulh(uint64_t a, uint64_t b) {
    const uint64_t m = (uint64_t)hi32(a) * lo32(b), n = (uint64_t)lo32(a) * hi32(b);
    return (uint64_t)hi32(a) * hi32(b) + hi32(m) + hi32(n);
}
// a b / 2^21, b of 21 bits.
__device__ __forceinline__ uint64_t mul21(uint64_t a, uint32_t b) {
    const uint64_t l = (uint64_t)lo32(a) * b, h = (uint64_t)hi32(a) * b + hi32(l);
    return (h << 11) | (lo32(l) >> 21);
}

// m 2^(e - 63) / 2^1023 rounded to nearest (0 < m < 2^63; e a biased exponent, of a leading one at bit 63).  WIDE: m may be
// below 2^32, and the value is 0 where it is below the normal range.
template <bool WIDE>
__device__ __forceinline__ double pack(uint64_t m, int e, uint32_t sign = 0) {
    const int z = WIDE ? __clzll((long long)m) : __clz((int)hi32(m));
    const int f = e - z - 1;   // (the leading one of the mantissa adds 1)
    const uint64_t b = ((m << (z - 1)) + 0x200) >> 10;
    const double v = __hiloint2double((int)(hi32(b) + ((uint32_t)f << 20) + (sign << 31)), (int)lo32(b));
    return WIDE && f < 0 ? 0.0 : v;
}

// y = the hardware approximation of 1/x (21 bits, 2^-19.9) and c = 1 / (x y) in Q63: with e = 1 - x y, exact in the low word
// of the product of the mantissas, 1 + e + e^2.  False where x is not positive and normal (y may be none).
__device__ __forceinline__ bool rcp21(double x, uint32_t& ym, int& ye, uint64_t& c) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const uint32_t xh = (uint32_t)__double2hiint(x), yh = (uint32_t)__double2hiint(y);
    ym = (yh & 0xFFFFF) | 0x100000;
    ye = (int)(yh >> 20);
    const int s = (int)(xh >> 20) + ye - 2046;   // 0 or -1: x y = product / 2^(72 - s)
    const uint64_t p = (uint64_t)(uint32_t)__double2loint(x) * ym + ((uint64_t)(((xh & 0xFFFFF) | 0x100000) * ym) << 32);
    const int64_t e = -(int64_t)(p << ((1 + s) & 1));   // in Q73
    const int eh = (int)(e >> 32);
    c = 0x8000000000000000ull + (uint64_t)((e + (((int64_t)eh * eh) >> 9)) >> 10);
    return (unsigned)(s + 1) <= 1u;
}

// y = the hardware approximation of 1/sqrt(x) (21 bits, 2^-19) and c = 1 / (y sqrt(x)) in Q63: 1 + e / 2 + 3 e^2 / 8 from the
// residual e = 1 - x y^2, x = xm 2^(xe - 1023 - 63).  False where x is not positive and normal.
__device__ __forceinline__ bool rsqrt21(double x, uint64_t xm, uint32_t& ym, int& xe, int& ye, uint64_t& c) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const uint32_t xh = (uint32_t)__double2hiint(x), yh = (uint32_t)__double2hiint(y);
    ym = (yh & 0xFFFFF) | 0x100000;
    xe = (int)(xh >> 20);
    ye = (int)(yh >> 20);
    const int s = xe + 2 * ye - 3069 + 2;   // 0 .. 2: x y^2 = product / 2^(63 - s)
    const int64_t r = (int64_t)(0x8000000000000000ull - (mulh(xm, ((uint64_t)ym * ym) << 22) << (s & 3)));   // e in Q63
    const int e49 = (int)(r >> 14);
    const uint64_t q = (uint64_t)((int64_t)e49 * e49) >> 35;   // e^2 in Q63
    c = 0x8000000000000000ull + (uint64_t)(r >> 1) + ((3 * q) >> 3);
    return (unsigned)s <= 2u;
}

// sqrt(x) (x > 0), to nearest up to 2^-59.
__device__ __forceinline__ double sqrt64(double x) {
    uint32_t ym;
    int xe, ye;
    uint64_t c;
    const uint64_t xm = mant(x);
    return rsqrt21(x, xm, ym, xe, ye, c) ? pack<false>(mulh(c, mul21(xm, ym)), xe + ye - 1023 + 2) : sqrt(x);
}

// 1 / sqrt(x) (x > 0), to nearest up to 2^-58, and in wy w times it, w of mantissa wm and biased exponent we.
__device__ __forceinline__ double rsqrt64(double x, uint64_t wm, int we, double w, double& wy) {
    uint32_t ym;
    int xe, ye;
    uint64_t c;
    const bool ok = rsqrt21(x, mant(x), ym, xe, ye, c);
    const uint64_t m = mul21(c, ym);
    double y = pack<false>(m, ye + 1);
    wy = pack<false>(mulh(m, wm), ye + 1 + we - 1023 + 1);
    if (__any_sync(__activemask(), !ok)) {
        const double l = 1.0 / sqrt(x);
        y = ok ? y : l;
        wy = ok ? wy : w * l;
    }
    return y;
}

// Vectors in block fixed point: component = (h 2^30 + l) 2^(E - 60), |h| <= 2^30, |l| <= 2^29, one E per vector.
__device__ __forceinline__ int2 limbs(int64_t i) {
    const int l = (int)(((uint32_t)i + (1u << 29)) & 0x3FFFFFFFu) - (1 << 29);
    return make_int2((int)((i - l) >> 30), l);
}
// x 2^(60 - E), to nearest, down = E - 1 minus the exponent of x (not negative).
__device__ __forceinline__ int64_t fix60(double x, int down) {
    const int64_t m = down > 59 ? 0 : (int64_t)(((mant(x) >> (3 + down)) + 1) >> 1);
    return __double2hiint(x) < 0 ? -m : m;
}
// The inner product of two such vectors / 2^(E + E' - 60): nine 32-bit products (the product of the low limbs, below a unit,
// is left out).
__device__ __forceinline__ int64_t dot60(int2 ax, int2 ay, int2 az, int2 bx, int2 by, int2 bz) {
    const int64_t mid = (int64_t)ax.x * bx.y + (int64_t)ax.y * bx.x + (int64_t)ay.x * by.y + (int64_t)ay.y * by.x +
                        (int64_t)az.x * bz.y + (int64_t)az.y * bz.x + (1 << 29);
    return (int64_t)ax.x * bx.x + (int64_t)ay.x * by.x + (int64_t)az.x * bz.x + (mid >> 30);
}
// r 2^(e - 60), rounded to nearest.
__device__ __forceinline__ double value60(int64_t r, int e) {
    const uint64_t m = (uint64_t)(r < 0 ? -r : r);
    return pack<true>(m | 1, m ? e + 1026 : 0, (uint32_t)((uint64_t)r >> 63));
}

// 1 / sqrt(n) and w / sqrt(n), n = |r|^2 of r in block fixed point (h 2^30 + l with 0 <= l < 2^30, below 2^60; exponent E).
// False where |r| < 2^(E - 6), for which 60 bits of r are too few, or |r| = 0.
__device__ __forceinline__ bool rnorm60(const int2 r[3], int E, uint64_t wm, int we, double& y, double& wy) {
    const int64_t hh = (int64_t)r[0].x * r[0].x + (int64_t)r[1].x * r[1].x + (int64_t)r[2].x * r[2].x;
    const int64_t hl = (int64_t)r[0].x * r[0].y + (int64_t)r[1].x * r[1].y + (int64_t)r[2].x * r[2].y;
    const int64_t ll = (int64_t)r[0].y * r[0].y + (int64_t)r[1].y * r[1].y + (int64_t)r[2].y * r[2].y;
    const int z = max(__clz((int)hi32((uint64_t)hh)) - 2, 0);   // n 2^60 2^(-2 E) in Q(z): s < 2^63
    const uint64_t s = ((uint64_t)hh << z) + (uint64_t)(hl >> (29 - min(z, 29))) + (uint64_t)(ll >> (60 - z));
    const int up = __clz((int)hi32(s));
    const uint64_t m = s << up;
    // n = m 2^-63 2^x, x = 2 E + 3 - z - up
    const int odd = (z + up + 1) & 1, xh = 2 * E + 3 - z - up - odd;
    uint32_t ym;
    int xe, ye;
    uint64_t c;
    rsqrt21(__hiloint2double((int)(((1022 + odd) << 20) + (int)(m >> 43)), (int)(m >> 11)), m, ym, xe, ye, c);
    const uint64_t q = mul21(c, ym);
    const int e = ye + 1 - xh / 2;
    y = pack<false>(q, e);
    wy = pack<false>(mulh(q, wm), e + we - 1022);
    return z <= 10;
}

// atanh(z) / z - 1 of z in Q64 below 1/2, Q64: w f(w), w = z^2, f by the polynomial that interpolates it at the Chebyshev
// nodes of [0, 1/4] (2^-66.7), in v = 1 - 4 w, where its terms alternate and every partial sum is positive.
__device__ __forceinline__ uint64_t atanh_half(uint64_t z) {
    const uint64_t w = mulh(z, z) << 2, v = 0 - w;
    uint64_t a = 0x2be0df598ull - mulh(v, 0x3e8948b0ull);
    a = 0xff24812e9ull - mulh(v, a);
    a = 0x430d9773b0ull - mulh(v, a);
    a = 0xf06b94e6daull - mulh(v, a);
    a = 0x3293677c076ull - mulh(v, a);
    a = 0xa7bb1d7e58full - mulh(v, a);
    a = 0x22e9cd7f3608ull - mulh(v, a);
    a = 0x758d87dfb77bull - mulh(v, a);
    a = 0x191b478a962e7ull - mulh(v, a);
    a = 0x57780fd68e50cull - mulh(v, a);
    a = 0x138c45ddaf52f7ull - mulh(v, a);
    a = 0x4885c5685f8e9full - mulh(v, a);
    a = 0x11c96d20d77958full - mulh(v, a);
    a = 0x4ccaf2a7261ac2bull - mulh(v, a);
    a = 0x193ea7aad030a976ull - mulh(v, a);
    return mulh(w, a);
}

// 2 atanh(len / R) / len = log((R + len) / (R - len)) / len (times the weight of mantissa wm and biased exponent we where
// WEIGHT), 0 < len < R.  With z = len / R: 2 / R (1 + u), u = atanh(z) / z - 1, by polynomials on [0, 1/8] (2^-65) and
// [0, 1/4] (2^-67) or atanh_half.  From z = 1/2 on, with a = R + len and b = R - len (exact): (k log 2 + 2 atanh((a - 2^k b) / (a + 2^k b))) / len,
// k the difference of their exponents, so that the quotient is below 1/3.
template <bool WEIGHT>
__device__ __forceinline__ double edge(double R, double len, uint64_t wm, int we, double wr) {
    uint32_t ym;
    int ye;
    uint64_t c;
    const bool ok = rcp21(R, ym, ye, c);
    const int sh = 2044 - (int)expo(len) - ye;
    uint64_t z = (mulh(mul21(mant(len), ym), c) << 1) >> min(max(sh, 0), 63);   // Q64
    const bool direct = ok && sh >= 0 && z < (1ull << 63);
    const unsigned lanes = __activemask();   // one polynomial for the whole warp, and FP64 in the rare branch alone
    uint64_t u;
    if (__all_sync(lanes, direct && z < (1ull << 61))) {
        const uint64_t w = mulh(z, z) << 6;
        const uint32_t wh = hi32(w);
        uint32_t t = __umulhi(wh, 0x47a94u) + 0x13ac84au;
        t = __umulhi(wh, t) + 0x5d177978u;
        u = 0x1c71c70a52ull + __umulhi(wh, t);
        u = 0x92492492799ull + mulh(u, w);
        u = 0x3333333333303ull + mulh(u, w);
        u = 0x155555555555556ull + mulh(u, w);
        u = mulh(u, w);
    } else if (__all_sync(lanes, direct && z < (1ull << 62))) {
        const uint64_t w = mulh(z, z) << 4;
        const uint32_t wh = hi32(w);
        uint32_t t = __umulhi(wh, 0x105317u) + 0xce4dedu;
        t = __umulhi(wh, t) + 0xf1a4366u;
        u = 0x11108fa10ull + __umulhi(wh, t);
        u = 0x13b13eabf7ull + mulh(u, w);
        u = 0x1745d164db2ull + mulh(u, w);
        u = 0x1c71c71c981eull + mulh(u, w);
        u = 0x2492492492191ull + mulh(u, w);
        u = 0x3333333333334bull + mulh(u, w);
        u = 0x555555555555555ull + mulh(u, w);
        u = mulh(u, w);
    } else {
        int k = 0;
        uint32_t minus = 0;
        bool none = false;
        const bool far = __all_sync(lanes, direct);
        if (!far) {
            const double a = R + len, b = R - len;
            const int kk = (int)expo(a) - (int)expo(b);
            const double bk = __hiloint2double(__double2hiint(b) + (kk << 20), __double2loint(b));
            const double n = a - bk, d = a + bk;
            uint32_t dm;
            int de;
            uint64_t dc;
            none = !(rcp21(d, dm, de, dc) && __double2hiint(b) > 0x100000 && expo(a) < 0x7FE && (unsigned)kk < 64u && expo(len) != 0);
            if (!direct) {
                k = kk;
                minus = (uint32_t)__double2hiint(n) >> 31;
                z = expo(n) ? (mulh(mul21(mant(n), dm), dc) << 1) >> min(max(2044 - (int)expo(n) - de, 0), 63) : 0;
            }
        }
        u = atanh_half(z);
        if (!direct) {
            if (none) return (WEIGHT ? wr : 1.0) * (log((R + len) / (R - len)) / len);
            const uint64_t t = mulh(z, 0x8000000000000000ull + (u >> 1)) >> 5;   // 2 atanh in Q57
            const uint64_t base = 0x162E42FEFA39EF3ull * (uint64_t)k;            // k log 2 in Q57
            const uint64_t sum = minus ? base - t : base + t;
            const int zs = __clzll((long long)(sum | 1));
            rcp21(len, ym, ye, c);
            uint64_t m = mulh(sum << zs, c);
            if (WEIGHT) m = mulh(m, wm);
            return pack<false>(mul21(m, ym), (WEIGHT ? we - 1023 + 1 : 0) + ye + 8 - zs);
        }
    }
    uint64_t m = mulh(0x8000000000000000ull + (u >> 1), c);
    if (WEIGHT) m = mulh(m, wm);
    return pack<false>(mul21(m, ym), (WEIGHT ? we - 1023 + 1 : 0) + ye + 3);
}

// atan2(num, den), half a solid angle (times the weight where WEIGHT).  Where t = num / den < 1/2 and den > 0:
// t (1 - w g(w)), w = t^2, g interpolated on [0, 2^-8], [0, 2^-4] and [0, 1/4] (2^-70, 2^-61.8 and 2^-64).  Elsewhere the angle
// from the nearest of pi/4, pi/2, 3 pi/4 and pi, whose tangent is below 1/2.
template <bool WEIGHT>
__device__ __forceinline__ double half_angle(double num, double den, uint64_t wm, int we, double wr) {
    uint32_t ym;
    int ye;
    uint64_t c;
    const bool ok = rcp21(den, ym, ye, c);
    int ne = (int)expo(num), sh = 2044 - ne - ye;
    uint64_t q = mulh(mul21(mant(num), ym), c) << 1;   // the quotient's mantissa in Q62
    uint64_t t = q >> min(max(sh, 0), 63);
    const bool direct = ok && sh >= 0 && t < (1ull << 63);
    const unsigned lanes = __activemask();
    uint32_t sign = (uint32_t)__double2hiint(num) >> 31;
    uint64_t u;
    if (__all_sync(lanes, direct && t < (1ull << 60))) {
        const uint64_t w = mulh(t, t) << 8;
        const uint32_t wh = hi32(w);
        uint32_t a = 0x174598u - __umulhi(wh, 0x137eu);
        a = 0x1c71c6ffu - __umulhi(wh, a);
        u = 0x249249248bull - __umulhi(wh, a);
        u = 0x333333333333ull - mulh(u, w);
        u = 0x55555555555555ull - mulh(u, w);
        u = mulh(u, w);
    } else if (__all_sync(lanes, direct && t < (1ull << 62))) {
        const uint64_t w = mulh(t, t) << 4;
        const uint32_t wh = hi32(w);
        const uint32_t a = 0xeba484cu - __umulhi(wh, 0xa8138cu);
        u = 0x110bd65edull - __umulhi(wh, a);
        u = 0x13b10a743bull - mulh(u, w);
        u = 0x1745d069642ull - mulh(u, w);
        u = 0x1c71c71937c7ull - mulh(u, w);
        u = 0x249249248d464ull - mulh(u, w);
        u = 0x33333333333033ull - mulh(u, w);
        u = 0x555555555555551ull - mulh(u, w);
        u = mulh(u, w);
    } else {
        double base = 0.0;
        bool none = false;
        const bool far = __all_sync(lanes, direct);
        if (!far) {
            const double an = fabs(num), ad = fabs(den);
            const long long in = __double_as_longlong(an), id = __double_as_longlong(ad), one = 1ll << 52;
            const bool left = __double2hiint(den) < 0;
            const double dif = an - ad, sum = an + ad;
            double n, d;
            if (in > id + one) {   // |num| > 2 |den|: from pi/2
                base = 1.5707963267948966;
                n = -den;
                d = an;
            } else if (in + one > id) {   // from pi/4 or 3 pi/4
                base = left ? 2.356194490192345 : 0.7853981633974483;
                n = left ? -dif : dif;
                d = sum;
            } else {   // from pi (num < den / 2 with den > 0 is direct, or not finite)
                base = 3.141592653589793;
                n = -an;
                d = ad;
            }
            const long long big = in > id ? in : id;
            uint32_t dm;
            int de;
            uint64_t dc;
            none = !(rcp21(d, dm, de, dc) && big >= (one << 1) && big < 0x7FD0000000000000ll && (left || in + one > id));
            if (!direct) {
                base = sign ? -base : base;
                sign ^= (uint32_t)__double2hiint(n) >> 31;
                ne = (int)expo(n);
                ye = de;
                q = mulh(mul21(mant(n), dm), dc) << 1;
                t = q >> min(max(2044 - ne - de, 0), 63);
            }
        }
        const uint64_t w = mulh(t, t) << 2;
        uint64_t a = 0x1633de284ull - mulh(w, 0x1f5c3523ull);
        a = 0x8b3543996ull - mulh(w, a);
        a = 0x2ad65f05c0ull - mulh(w, a);
        a = 0xc1bd2924cfull - mulh(w, a);
        a = 0x35d96a84825ull - mulh(w, a);
        a = 0xf0ec54dd6c3ull - mulh(w, a);
        a = 0x44442fbedc95ull - mulh(w, a);
        a = 0x13b13ad5571f0ull - mulh(w, a);
        a = 0x5d1745c9c07a2ull - mulh(w, a);
        a = 0x1c71c71c68a0c5ull - mulh(w, a);
        a = 0x9249249248c994ull - mulh(w, a);
        a = 0x3333333333331ceull - mulh(w, a);
        a = 0x1555555555555554ull - mulh(w, a);
        u = mulh(w, a);
        if (!far) {
            const double v = pack<true>(mulh(0x8000000000000000ull - (u >> 1), q) | 1, ne ? ne + ye - 1023 + 2 : 0, sign) + base;
            const double x = none ? atan2(num, den) : v;
            if (!direct) return WEIGHT ? wr * x : x;
        }
    }
    uint64_t m = mulh(0x8000000000000000ull - (u >> 1), q);
    if (WEIGHT) m = mulh(m, wm);
    return pack<true>(m | 1, ne ? (WEIGHT ? we - 1023 + 1 : 0) + ne + ye - 1023 + 2 : 0, sign);
}

}  // namespace fx
}  // namespace omg
