// Roots and distances shared by the pair kernels, and the factorization's reciprocal.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace tpe {

// 1/sqrt(x) for normal x > 0: the hardware's approximation y (20 bits) corrected by the
// binomial series of (1 - e)^(-1/2), e = 1 - x y^2, through e^2 (|e| is below 2^-19, the
// 5/16 e^3 left out below 2^-58). Zero, subnormal, infinite and NaN x give infinity or
// NaN: the callers test for what they accept. Largest error in a million samples 1.24
// units of 2^-53, root mean square 0.48 (CUDA's rsqrt, which branches: 1.00 and 0.43).
__device__ __forceinline__ double rsqrt_normal(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// 1/x for normal x whose reciprocal is normal: the hardware's approximation y (20 bits)
// times the geometric series of 1/(1 - e), e = 1 - x y, through e^2 (the e^3 left out is
// below 2^-57). Largest error 1.002 units of 2^-53; the division's is 1, and takes 2.5 us
// more per 64 columns of the factorization.
__device__ __forceinline__ double recip_normal(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// x^(-1/3): an FP32 estimate y (exp2 of log2) times the binomial series of
// (1 - e)^(-1/3), e = 1 - x y^3, through e^3. The estimate is 1e-7 off at x = 1 and 3e-6
// where |log2 x| is 100 (the rounding of a logarithm of that size), so that the e^4 left out
// is below 2^-66. false (r is then of no use) beyond the range where FP32 holds y and y^3.
// Largest error in a million samples 1.16 units of 2^-53 from 1e-30 to 1e30 (1.36 at its ends
// without the e^3 term, which costs no time that shows); rcbrt 1.00.
__device__ __forceinline__ bool inv_cbrt_fast(double x, double& r) {
    const double y = (double)exp2f(-0.33333334f * __log2f((float)x));
    const double e = fma(-x * y, y * y, 1.0);
    r = fma(y * e, fma(fma(14.0 / 81.0, e, 2.0 / 9.0), e, 1.0 / 3.0), y);
    return x > 1e-30 && x < 1e30;
}
// The same for any x > 0: CUDA's own beyond that range.
__device__ __forceinline__ double inv_cbrt(double x) {
    double r;
    return inv_cbrt_fast(x, r) ? r : rcbrt(x);
}

// r = 1/sqrt(x) and inv_se = 1/(sqrt(x) + eps) = r / (1 + t) with t = eps r, summed as
// r (1 - t + t^2): the first term left out is below 2^-60 relative for t < 2^-20. false
// (neither is then of use) for larger t, distances within about 1e6 eps of zero, and for
// zero, subnormal and non-finite x.
__device__ __forceinline__ bool inv_dist_fast(double x, double eps, double& r, double& inv_se) {
    r = rsqrt_normal(x);
    const double t = eps * r;
    inv_se = fma(-r, t * (1.0 - t), r);
    return t < 9.5367431640625e-07;
}

// s = sqrt(x), inv_s = 1/s (0 below 1e-14) and inv_se = 1/(s + eps) for x >= 0, from one
// reciprocal square root where inv_dist_fast holds, else from the square root and divisions.
__device__ __forceinline__ void dist_terms(double x, double eps, double& s, double& inv_s,
                                           double& inv_se) {
    double r;
    if (inv_dist_fast(x, eps, r, inv_se)) {
        s = x * r;
        inv_s = r;
    } else {
        s = sqrt(x);
        inv_s = s < 1e-14 ? 0.0 : 1.0 / s;
        inv_se = 1.0 / (s + eps);
    }
}

__device__ __forceinline__ bool disjoint(int2 a, int2 b) {
    return a.x != b.x && a.x != b.y && a.y != b.x && a.y != b.y;
}

}  // namespace tpe
