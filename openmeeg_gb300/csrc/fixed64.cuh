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

// 2 atanh(len / R) / len (times the weight of mantissa wm and biased exponent we where WEIGHT), 0 < len < R: with z = len / R
// and w = z^2, 2 / R (1 + u), u = w f(w) = atanh(z) / z - 1 by the polynomials that interpolate f at the Chebyshev nodes of
// [0, 2^-6] and [0, 1/4] (relative error of the result 2^-65 and 2^-62.8), the library's logarithm beyond z = 1/2.
template <bool WEIGHT>
__device__ __forceinline__ double edge(double R, double len, uint64_t wm, int we, double wr) {
    uint32_t ym;
    int ye;
    uint64_t c;
    const bool ok = rcp21(R, ym, ye, c);
    const int sh = 2044 - (int)expo(len) - ye;
    const uint64_t z = (mulh(mul21(mant(len), ym), c) << 1) >> min(max(sh, 0), 63);   // Q64
    uint64_t w = mulh(z, z), u;
    if (__all_sync(__activemask(), ok && sh >= 0 && z < (1ull << 61))) {   // (one polynomial for the whole warp)
        w <<= 6;
        const uint32_t wh = hi32(w);
        uint32_t t = __umulhi(wh, 0x47a94u) + 0x13ac84au;
        t = __umulhi(wh, t) + 0x5d177978u;
        u = 0x1c71c70a52ull + __umulhi(wh, t);
        u = 0x92492492799ull + mulh(u, w);
        u = 0x3333333333303ull + mulh(u, w);
        u = 0x155555555555556ull + mulh(u, w);
        u = mulh(u, w);
    } else if (ok && sh >= 0 && z < (1ull << 63)) {
        const int64_t v = (int64_t)(w << 1);   // w / (1/4) in Q63
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
        u = (uint64_t)(__mul64hi(v, a) << 1);
    } else {
        const double l = log((R + len) / (R - len)) / len;
        return WEIGHT ? l * wr : l;
    }
    uint64_t m = mulh(0x8000000000000000ull + (u >> 1), c);
    if (WEIGHT) m = mulh(m, wm);
    return pack(mul21(m, ym), (WEIGHT ? we - 1023 + 1 : 0) + ye + 3);
}

// atan2(num, den), half a solid angle (times the weight where WEIGHT): where t = num / den < 1/2 and den > 0 by
// t (1 - w g(w)), w = t^2, g interpolated on [0, 2^-8] and [0, 1/4] (relative error of the result 2^-70 and 2^-64).
template <bool WEIGHT>
__device__ __forceinline__ double half_angle(double num, double den, uint64_t wm, int we, double wr) {
    uint32_t ym;
    int ye;
    uint64_t c;
    const bool ok = rcp21(den, ym, ye, c);
    const int ne = (int)expo(num), sh = 2044 - ne - ye;
    const uint64_t q = mulh(mul21(mant(num), ym), c) << 1;   // the quotient's mantissa in Q62
    const uint64_t t = q >> min(max(sh, 0), 63);
    uint64_t w = mulh(t, t), u;
    if (__all_sync(__activemask(), ok && sh >= 0 && t < (1ull << 60))) {
        w <<= 8;
        const uint32_t wh = hi32(w);
        uint32_t a = 0x174598u - __umulhi(wh, 0x137eu);
        a = 0x1c71c6ffu - __umulhi(wh, a);
        u = 0x249249248bull - __umulhi(wh, a);
        u = 0x333333333333ull - mulh(u, w);
        u = 0x55555555555555ull - mulh(u, w);
        u = mulh(u, w);
    } else if (ok && sh >= 0 && t < (1ull << 63)) {
        w <<= 2;
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
    } else {
        const double v = atan2(num, den);
        return WEIGHT ? v * wr : v;
    }
    uint64_t m = mulh(0x8000000000000000ull - (u >> 1), q);
    if (WEIGHT) m = mulh(m, wm);
    return pack(m, ne ? (WEIGHT ? we - 1023 + 1 : 0) + ne + ye - 1023 + 2 : 0, (uint32_t)__double2hiint(num) >> 31);
}

}  // namespace fx
}  // namespace omg
