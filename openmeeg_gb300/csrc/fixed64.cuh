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

// m 2^(e - 63) / 2^1023 rounded to nearest (m != 0; e a biased exponent, of a leading one at bit 63); 0 where it is
// below the normal range.
__device__ __forceinline__ double pack(uint64_t m, int e, uint32_t sign = 0) {
    const int z = __clzll((long long)m);
    m <<= z;
    const int f = e - z;
    const uint64_t b = ((uint64_t)(uint32_t)(f - 1) << 52) + (m >> 11) + ((m >> 10) & 1);
    return f < 1 ? 0.0 : __longlong_as_double((long long)(b | ((uint64_t)sign << 63)));
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

// sqrt(x) (x > 0), to nearest up to 2^-59.
__device__ __forceinline__ double sqrt64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const uint32_t xh = (uint32_t)__double2hiint(x), yh = (uint32_t)__double2hiint(y);
    const uint32_t ym = (yh & 0xFFFFF) | 0x100000;
    const int xe = (int)(xh >> 20), ye = (int)(yh >> 20);
    const int s = xe + 2 * ye - 3069 + 2;   // 0 .. 2: x y^2 = product / 2^(63 - s)
    if ((unsigned)s > 2u) return sqrt(x);
    const uint64_t xm = mant(x);
    const int64_t e = (int64_t)(0x8000000000000000ull - (mulh(xm, ((uint64_t)ym * ym) << 22) << s));   // 1 - x y^2 in Q63
    const int e49 = (int)(e >> 14);
    const uint64_t q = (uint64_t)((int64_t)e49 * e49) >> 35;   // e^2 in Q63
    const uint64_t m = 0x8000000000000000ull + (uint64_t)(e >> 1) + ((3 * q) >> 3);   // 1 + e / 2 + 3 e^2 / 8
    const uint64_t g = mul21(xm, ym);   // x y = g 2^(xe - 1023 + ye - 1023 - 62)
    return pack(mulh(m, g), xe + ye - 1023 + 2);
}

// atanh(z) / z - 1 of z in Q64 below 1/2, Q64: w f(w), w = z^2, f by the polynomial that interpolates it at the Chebyshev
// nodes of [0, 1/4] (2^-62.8).
__device__ __forceinline__ uint64_t atanh_half(uint64_t z) {
    const int64_t v = (int64_t)(mulh(z, z) << 1);   // w / (1/4) in Q63
    int64_t a = -0x2f3bcdad3ll + (__mul64hi(v, 0xe7f9933cll) << 1);
    a = 0xa798b13acll + (__mul64hi(v, a) << 1);
    a = -0x17b097a15ll + (__mul64hi(v, a) << 1);
    a = 0x37febab086ll + (__mul64hi(v, a) << 1);
    a = 0xbb2926705bll + (__mul64hi(v, a) << 1);
    a = 0x3622dd23e5cll + (__mul64hi(v, a) << 1);
    a = 0xf0db60f9e55ll + (__mul64hi(v, a) << 1);
    a = 0x444498cb9d98ll + (__mul64hi(v, a) << 1);
    a = 0x13b13a3184d91ll + (__mul64hi(v, a) << 1);
    a = 0x5d1745ea0cee5ll + (__mul64hi(v, a) << 1);
    a = 0x1c71c71c58156bll + (__mul64hi(v, a) << 1);
    a = 0x924924924a04e3ll + (__mul64hi(v, a) << 1);
    a = 0x333333333333030ll + (__mul64hi(v, a) << 1);
    a = 0x1555555555555557ll + (__mul64hi(v, a) << 1);
    return (uint64_t)(__mul64hi(v, a) << 1);
}

// 2 atanh(len / R) / len = log((R + len) / (R - len)) / len (times the weight of mantissa wm and biased exponent we where
// WEIGHT), 0 < len < R.  With z = len / R: 2 / R (1 + u), u = atanh(z) / z - 1, by a polynomial on [0, 1/8] (2^-65) or
// atanh_half.  From z = 1/2 on, with a = R + len and b = R - len (exact): (k log 2 + 2 atanh((a - 2^k b) / (a + 2^k b))) / len,
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
    uint64_t u;
    if (__all_sync(__activemask(), direct && z < (1ull << 61))) {   // (one polynomial for the whole warp)
        const uint64_t w = mulh(z, z) << 6;
        const uint32_t wh = hi32(w);
        uint32_t t = __umulhi(wh, 0x47a94u) + 0x13ac84au;
        t = __umulhi(wh, t) + 0x5d177978u;
        u = 0x1c71c70a52ull + __umulhi(wh, t);
        u = 0x92492492799ull + mulh(u, w);
        u = 0x3333333333303ull + mulh(u, w);
        u = 0x155555555555556ull + mulh(u, w);
        u = mulh(u, w);
    } else {
        int k = 0;
        uint32_t minus = 0;
        if (!direct) {
            const double a = R + len, b = R - len;
            k = (int)expo(a) - (int)expo(b);
            const double bk = __hiloint2double(__double2hiint(b) + (k << 20), __double2loint(b));
            const double n = a - bk, d = a + bk;
            uint32_t dm;
            int de;
            uint64_t dc;
            if (!(__double2hiint(b) > 0x100000 && expo(a) < 0x7FE && (unsigned)k < 64u && rcp21(d, dm, de, dc) && expo(len) != 0))
                return (WEIGHT ? wr : 1.0) * (log((R + len) / (R - len)) / len);
            minus = (uint32_t)__double2hiint(n) >> 31;
            const int s = 2044 - (int)expo(n) - de;
            z = expo(n) ? (mulh(mul21(mant(n), dm), dc) << 1) >> min(max(s, 0), 63) : 0;
        }
        u = atanh_half(z);
        if (!direct) {
            const uint64_t t = mulh(z, 0x8000000000000000ull + (u >> 1)) >> 5;   // 2 atanh in Q57
            const uint64_t base = 0x162E42FEFA39EF3ull * (uint64_t)k;            // k log 2 in Q57
            const uint64_t sum = minus ? base - t : base + t;
            const int zs = __clzll((long long)sum);
            rcp21(len, ym, ye, c);
            uint64_t m = mulh(sum << zs, c);
            if (WEIGHT) m = mulh(m, wm);
            // sum 2^-57 / len: m = sum 2^zs / 2 (/ 2), mul21 another 2^-21 of ym 2^20
            return pack(mul21(m, ym), (WEIGHT ? we - 1023 + 1 : 0) + ye + 8 - zs);
        }
    }
    uint64_t m = mulh(0x8000000000000000ull + (u >> 1), c);
    if (WEIGHT) m = mulh(m, wm);
    return pack(mul21(m, ym), (WEIGHT ? we - 1023 + 1 : 0) + ye + 3);
}

// atan2(num, den), half a solid angle (times the weight where WEIGHT).  Where t = num / den < 1/2 and den > 0:
// t (1 - w g(w)), w = t^2, g interpolated on [0, 2^-8] and [0, 1/4] (2^-70 and 2^-64).  Elsewhere the angle from the nearest of
// pi/4, pi/2, 3 pi/4 and pi, whose tangent is below 1/2.
template <bool WEIGHT>
__device__ __forceinline__ double half_angle(double num, double den, uint64_t wm, int we, double wr) {
    uint32_t ym;
    int ye;
    uint64_t c;
    bool ok = rcp21(den, ym, ye, c);
    int ne = (int)expo(num), sh = 2044 - ne - ye;
    uint64_t q = mulh(mul21(mant(num), ym), c) << 1;   // the quotient's mantissa in Q62
    uint64_t t = q >> min(max(sh, 0), 63);
    const bool direct = ok && sh >= 0 && t < (1ull << 63);
    uint32_t sign = (uint32_t)__double2hiint(num) >> 31;
    double base = 0.0;
    uint64_t u;
    if (__all_sync(__activemask(), direct && t < (1ull << 60))) {
        const uint64_t w = mulh(t, t) << 8;
        const uint32_t wh = hi32(w);
        uint32_t a = 0x174598u - __umulhi(wh, 0x137eu);
        a = 0x1c71c6ffu - __umulhi(wh, a);
        u = 0x249249248bull - __umulhi(wh, a);
        u = 0x333333333333ull - mulh(u, w);
        u = 0x55555555555555ull - mulh(u, w);
        u = mulh(u, w);
    } else {
        if (!direct) {
            const double an = fabs(num), ad = fabs(den);
            const long long in = __double_as_longlong(an), id = __double_as_longlong(ad), one = 1ll << 52;
            const bool left = __double2hiint(den) < 0;
            double n, d;
            if (in > id + one) {   // |num| > 2 |den|: from pi/2
                base = 1.5707963267948966;
                n = -den;
                d = an;
            } else if (in + one > id) {   // from pi/4 or 3 pi/4
                base = left ? 2.356194490192345 : 0.7853981633974483;
                n = an - ad;
                d = an + ad;
                n = left ? -n : n;
            } else {   // from pi (num < den / 2 with den > 0 is direct, or not finite)
                base = 3.141592653589793;
                n = -an;
                d = ad;
            }
            const long long big = in > id ? in : id;
            ok = rcp21(d, ym, ye, c) && big >= (one << 1) && big < 0x7FD0000000000000ll && (left || in + one > id);
            if (!ok) return (WEIGHT ? wr : 1.0) * atan2(num, den);
            base = sign ? -base : base;
            sign ^= (uint32_t)__double2hiint(n) >> 31;
            ne = (int)expo(n);
            sh = 2044 - ne - ye;
            q = mulh(mul21(mant(n), ym), c) << 1;
            t = q >> min(max(sh, 0), 63);
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
    }
    uint64_t m = mulh(0x8000000000000000ull - (u >> 1), q);
    if (WEIGHT && direct) m = mulh(m, wm);
    const double v = pack(m, ne ? (WEIGHT && direct ? we - 1023 + 1 : 0) + ne + ye - 1023 + 2 : 0, sign);
    return direct ? v : (WEIGHT ? wr : 1.0) * (base + v);
}

}  // namespace fx
}  // namespace omg
