// SiLU in double for the rows of a chunk (k_dn_prep_seq); host and device, so that a test can hold it against the C library without a GPU.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

namespace rc {

// a / (1 + exp(-a)) to within 2^-50 of itself (2^-51.4 seen, with the C library's exp and a division 2^-51.5). exp(-a) = 2^n exp(r) with n the integer nearest to -a / ln 2: adding 1.5 2^52 leaves it in the low bits of the
// sum. The reduction is Cody and Waite's (Software Manual for the Elementary Functions, 1980, chapter 6): ln 2 in two parts, here 744261118 / 2^30, whose
// product with n is exact, and the rest. exp(r), |r| <= ln 2 / 2, is its Taylor polynomial of degree 13 (the remainder, r^14 / 14!, is below 2^-57). The reciprocal
// of d = 1 + exp(-a) is one of fp32 (y, off by at most 2^-22) corrected to y (1 + e + e^2), e = 1 - d y, which leaves e^3. With degree 10 and
// one Newton step, good to 2^-40, the kernel takes 65.1 us for 2048 tokens, with this 69.3 (events of some 3 us in both).
__host__ __device__ inline double silu_d(double a) {
    if (!(fabs(a) < 80.0)) return a / (1.0 + exp(-a));
    const double magic = 6755399441055744.0, t = fma(a, -1.4426950408889634, magic), n = t - magic;
    const double r = fma(n, 4.2009150726810846e-11, fma(n, -744261118.0 / 1073741824.0, -a));
    double p = 1.0 / 6227020800.0, two_n;
    p = fma(p, r, 1.0 / 479001600.0); p = fma(p, r, 1.0 / 39916800.0); p = fma(p, r, 1.0 / 3628800.0); p = fma(p, r, 1.0 / 362880.0); p = fma(p, r, 1.0 / 40320.0);
    p = fma(p, r, 1.0 / 5040.0); p = fma(p, r, 1.0 / 720.0); p = fma(p, r, 1.0 / 120.0); p = fma(p, r, 1.0 / 24.0); p = fma(p, r, 1.0 / 6.0);
    p = fma(p, r, 0.5); p = fma(p, r, 1.0); p = fma(p, r, 1.0);
#ifdef __CUDA_ARCH__
    two_n = __hiloint2double((__double2loint(t) + 1023) << 20, 0);
#else
    uint64_t bits;
    memcpy(&bits, &t, 8);
    bits = (uint64_t)(uint32_t)((int32_t)(uint32_t)bits + 1023) << 52;
    memcpy(&two_n, &bits, 8);
#endif
    const double d = fma(p, two_n, 1.0);
    double y = (double)(1.0f / (float)d);
    const double e = fma(-d, y, 1.0);
    y = fma(y, fma(e, e, e), y);
    return a * y;
}

}  // namespace rc
