// Fixed-point digits of FP64 values by integer arithmetic, shared by the kernels
// that cut operands for exact products on the bf16 tensor cores.
#pragma once

#include <stdint.h>

namespace omg {
namespace tcr {

// x 2^k rounded to the nearest integer (ties to even), exactly, by integer
// arithmetic on the bits of x (|x 2^k| < 2^62): the same value as
// __double2ll_rn(x * 2^k) without the FP64 pipe.
__device__ __forceinline__ long long scaled_rn(double x, int k) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int E = (int)((b >> 52) & 0x7FF);
    const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | (E ? (1ull << 52) : 0ull);
    const int sh = (E ? E : 1) - 1075 + k;   // |x 2^k| = m 2^sh
    unsigned long long q;
    if (sh >= 0) {
        q = m << sh;
    } else if (sh < -63) {
        q = 0;   // below 2^-11
    } else {
        // t = m >> (r - 1) keeps the half bit as its lowest bit; the bits below it are the sticky part:
        // round up when the half bit is set and (anything below it is set, or q is odd)
        const int r1 = -sh - 1;
        const unsigned long long t = m >> r1;
        const unsigned long long sticky = (m & ((1ull << r1) - 1ull)) != 0ull ? 1ull : 0ull;
        q = t >> 1;
        q += t & (sticky | q) & 1ull;
    }
    return (b >> 63) ? -(long long)q : (long long)q;
}

}  // namespace tcr
}  // namespace omg
