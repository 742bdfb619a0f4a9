// quotient.h -- quotients by a divisor whose reciprocal is at hand, by fused multiply-adds, with the division's bits.
//
// Markstein, IBM J. Res. Dev. 34, 1990: with r = RN(1/b) and a quotient q off by at most an ulp, q + r RN(a - q b)
// is RN(a / b), as long as the remainder a - q b is exact.  Compared with the division bit for bit, on the
// host and on the device, by tests/quotient_check.cpp.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define QHD __host__ __device__ __forceinline__
#else
#define QHD inline
#endif

namespace dasha {

QHD double fused(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
QHD float fused(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    return __fmaf_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
// the bits of |v| of a float, the high word of |v| of a double
QHD unsigned magnitude(float v) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(v) & 0x7fffffffu;
#else
    uint32_t u;
    std::memcpy(&u, &v, sizeof(u));
    return u & 0x7fffffffu;
#endif
}
QHD unsigned magnitude(double v) {
#ifdef __CUDA_ARCH__
    return (unsigned)__double2hiint(v) & 0x7fffffffu;
#else
    uint64_t u;
    std::memcpy(&u, &v, sizeof(u));
    return (unsigned)(u >> 32) & 0x7fffffffu;
#endif
}

QHD bool last_bit(float v) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(v) & 1u;
#else
    uint32_t u;
    std::memcpy(&u, &v, sizeof(u));
    return u & 1u;
#endif
}
QHD bool last_bit(double v) {
#ifdef __CUDA_ARCH__
    return __double2loint(v) & 1;
#else
    uint64_t u;
    std::memcpy(&u, &v, sizeof(u));
    return u & 1u;
#endif
}

// a / d for d = 3 or 6, r = RN(1 / d): a r is within an ulp of the quotient (RN(1/3) is off by a third of an ulp), so
// one remainder correction gives it.  A sixth may be subnormal and lie in the middle between two values, where
// the rounding of r decides wrongly: a reciprocal too small and one too large give the two
// neighbours there, and the even one is taken (elsewhere they agree, as the quotient is a sixth of a unit or more from
// the middle).  The sign is a's, that of a zero too; infinities and NaN are those of the product.  Without a branch: with
// the division behind one for these cases the FP64 RK update takes 188 registers, 168 so.
template <class T>
QHD T over(T a, T d, T r) {
    constexpr unsigned inf = sizeof(T) == 4 ? 0x7f800000u : 0x7ff00000u;
    constexpr T off = sizeof(T) == 4 ? T(0x1p-22) : T(0x1p-51);
    const T q = a * r, rem = fused(-q, d, a);
    T e;
    if (d == T(6)) {
        const T lo = fused(rem, r * (T(1) - off), q), hi = fused(rem, r * (T(1) + off), q);
        e = last_bit(lo) ? hi : lo;
    } else {
        e = fused(rem, r, q);
    }
    return magnitude(a) >= inf ? q : copysign(e, a);
}

// a / b, r = RN(1 / b)
QHD double div_by_steps(double a, double b, double r) {
    // the exponents of a and r within 2^+-650 and 2^+-300
    const unsigned ea = magnitude(a) >> 20, er = magnitude(r) >> 20;
    if (ea - 373u < 1300u && er - 723u < 600u) {
        double q = a * r;
        q = fused(fused(-q, b, a), r, q);
        return fused(fused(-q, b, a), r, q);
    }
    return a / b;
}

}  // namespace dasha
