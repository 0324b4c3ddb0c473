// Reciprocals of the factorisation's pivots (factor.cu).  Host code too, so that their errors can be checked where there is no
// GPU.
#pragma once
#include <math.h>
#include <string.h>

#ifdef __CUDACC__
#define GT_PIVOT_FN __host__ __device__ __forceinline__
#else
#define GT_PIVOT_FN inline
#endif

namespace gt {

GT_PIVOT_FN long long bits_of(double d) {
#ifdef __CUDA_ARCH__
    return __double_as_longlong(d);
#else
    long long b;
    memcpy(&b, &d, sizeof(b));
    return b;
#endif
}
GT_PIVOT_FN double of_bits(long long b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(b);
#else
    double d;
    memcpy(&d, &b, sizeof(d));
    return d;
#endif
}

// 1 / d for a normal d below 2^1022: an FP32 seed of the mantissa and two of Newton's steps r += r (1 - d r), within 1.01 x
// 2^-53 of the value.  (The compiler's division occupies the FP64 pipe, two operations a clock and SM, three times as long, on
// the pivots' chain.)
GT_PIVOT_FN double recip64(double d) {
    const long long bits = bits_of(d);
    const int e = (int)(bits >> 52) - 1023;
    const double m = of_bits((bits & 0xfffffffffffffll) | 0x3ff0000000000000ll);      // in [1, 2)
    double r = (double)(1.0f / (float)m);
    r = fma(r, fma(-m, r, 1.0), r);
    r = fma(r, fma(-m, r, 1.0), r);
    return r * of_bits((long long)(1023 - e) << 52);
}

// (re, im) = 1 / (re, im).  False, and the inverse of 1e-150, for a pivot whose squared magnitude is not above 1e-300 or not
// finite.  Where that square is 2^1022 or more, its reciprocal would be no normal number: it is taken of 2^-100 of the pivot.
GT_PIVOT_FN bool pivot_recip(double& re, double& im) {
    const double dd = re * re + im * im;
    if (dd > 1e-300 && dd < 0x1p1022) {
        const double r = recip64(dd);
        re *= r;
        im *= -r;
        return true;
    }
    if (dd > 1e-300 && dd <= 0x1.fffffffffffffp1023) {
        const double a = 0x1p-100 * re, b = 0x1p-100 * im, r = 0x1p-100 * recip64(a * a + b * b);
        re = a * r;
        im = -b * r;
        return true;
    }
    re = 1e150;
    im = 0.0;
    return false;
}

}  // namespace gt
