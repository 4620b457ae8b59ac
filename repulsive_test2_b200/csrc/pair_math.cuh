// Distance and power helpers shared by the pair kernels.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace tpe {

// 1/sqrt(x) for normal x > 0, to about one unit in the last place: the hardware's
// approximation y (20 bits) corrected by the binomial series of (1 - e)^(-1/2),
// e = 1 - x y^2, through e^2 (the e^3 left out is below 2^-60). Zero, subnormal,
// infinite and NaN x give infinity or NaN: the callers test for what they accept.
__device__ __forceinline__ double rsqrt_normal(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// s = sqrt(x), inv_s = 1/s (0 below 1e-14) and inv_se = 1/(s + eps) for x >= 0,
// from one reciprocal square root r: s = x r and 1/(s + eps) = r / (1 + t) with
// t = eps r, summed as r (1 - t + t^2) when t < 2^-20 (the first term left out
// is below 2^-60 relative). Distances within about 1e6 eps of zero (and
// non-finite input) take the square root and the divisions themselves.
__device__ __forceinline__ void dist_terms(double x, double eps, double& s, double& inv_s,
                                           double& inv_se) {
    const double r = rsqrt_normal(x);
    const double t = eps * r;
    if (t < 9.5367431640625e-07) {
        s = x * r;
        inv_s = r;
        inv_se = fma(-r, t * (1.0 - t), r);
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
