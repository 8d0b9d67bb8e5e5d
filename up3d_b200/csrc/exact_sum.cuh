// A sum of doubles that is the same for every order of its terms (host and
// device; no CUDA headers).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define UP3D_HD __host__ __device__ __forceinline__
#else
#define UP3D_HD inline
#endif

namespace up3d {

// Exponent field of a double: 0 for zero and subnormals, 2047 for infinities
// and NaN; the larger magnitude never has the smaller field.
UP3D_HD int exponent_field(double v) {
    uint64_t b;
    memcpy(&b, &v, sizeof b);
    return (int)(b >> 52 & 0x7ff);
}

// Terms are added as integers in units of 2^-95 of the power of two at or
// below the largest of them (`top`: its exponent field), each rounded to a
// unit where it has bits below, in 128 bits: room for 2^30 terms.  So n terms
// carry an error of at most n 2^-96 of the largest, and the result is that
// rounded to nearest once; the terms negated give the result negated.  With
// infinities or NaN among the terms the sum is theirs.
struct ExactSum {
    static constexpr int UNIT_BITS = 43;   // below the 53-bit significand of the largest
    __int128 sum = 0;
    double nonfinite = 0.0;
    int top;
    UP3D_HD explicit ExactSum(int top) : top(top) {}
    UP3D_HD void add(double v) {
        uint64_t b;
        memcpy(&b, &v, sizeof b);
        const int e = (int)(b >> 52 & 0x7ff);
        if (e == 0x7ff) nonfinite += v;
        uint64_t m = b & ((uint64_t(1) << 52) - 1);
        if (e) m |= uint64_t(1) << 52;
        const int shift = UNIT_BITS - ((top > 1 ? top : 1) - (e > 1 ? e : 1));
        __int128 term = 0;
        if (shift >= 0) term = (__int128)m << (shift < 64 ? shift : 64);
        else if (shift > -55) term = (__int128)((m + (uint64_t(1) << (-shift - 1))) >> -shift);
        sum += b >> 63 ? -term : term;
    }
    UP3D_HD double value() const {
        if (top == 0x7ff) return nonfinite;
        const unsigned __int128 m = sum < 0 ? -(unsigned __int128)sum : (unsigned __int128)sum;
        const uint64_t hi = (uint64_t)(m >> 64), lo = (uint64_t)m;
        int exponent = (top > 1 ? top : 1) - 1075 - UNIT_BITS;
        double r;
        if (hi == 0) {
            r = (double)lo;
        } else {   // the leading 64 bits, what is below them kept as a sticky bit
#ifdef __CUDA_ARCH__
            const int up = __clzll((long long)hi);
#else
            const int up = __builtin_clzll(hi);
#endif
            const unsigned __int128 s = m << up;
            r = (double)((uint64_t)(s >> 64) | ((uint64_t)s != 0));
            exponent += 64 - up;
        }
        r = ldexp(r, exponent);
        return sum < 0 ? -r : r;
    }
};

}  // namespace up3d
