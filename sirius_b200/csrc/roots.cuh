// roots.cuh — scalar roots of the step control and of the event location, for the device
// and, in host-only translation units, as plain host code.
#pragma once

#include "dual.cuh"

#ifdef __CUDACC__
#define SIRIUS_DEVICE __device__
#else
#define SIRIUS_DEVICE
#endif

namespace sirius {

// The zero in [0, 1] of the cubic Hermite interpolant of z over the accepted step
// (z0 and z1 have opposite signs): Newton from the chord's zero, kept inside the
// shrinking bracket (a step that leaves it bisects), to FP64 rounding, where bisection to
// the same width takes 60 iterations. Convergence is tested on the correction, before the
// bracket: the iterate has just become one of the bracket's ends, and a correction that
// rounds to zero would not lie inside. End slopes within 10 % of the chord's take 3.5 iterations in
// the mean and at most 4, within a factor of 2 to 3 4.4 and at most 6.
SIRIUS_DEVICE __forceinline__ double hermite_root(double z0, double z1, double dz0, double dz1, double h,
                                              int* iterations = nullptr) {
    const double m0 = mul_(h, dz0), m1 = mul_(h, dz1), d = z1 - z0;
    const double c2 = fma_(3.0, d, fma_(-2.0, m0, -m1)), c3 = fma_(-2.0, d, m0 + m1);
    double lo = 0.0, hi = 1.0, s = -z0 / d;
    int it = 0;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    while (it < 60) {
        ++it;
        const double f = fma_(s, fma_(s, fma_(s, c3, c2), m0), z0);
        const double df = fma_(s, fma_(s, mul_(3.0, c3), mul_(2.0, c2)), m0);
        const double t = s - f / df;
        if (fabs(t - s) < 1e-15) {
            s = t;
            break;
        }
        if ((f < 0.0) == (z0 < 0.0)) lo = s;
        else hi = s;
        s = t > lo && t < hi ? t : 0.5 * (lo + hi);
        if (hi - lo < 1e-15) break;
    }
    if (iterations) *iterations = it;
    return s;
}

// e^(-1/5) of e > 0: an FP32 estimate from the hardware logarithm and exponential
// (1e-5 relative at worst), and two Newton steps of y -> y + y (1 - e y^5) / 5, whose
// error goes from d to 3 d^2: FP64 rounding after the second (1.8e-16 over 1e-15..1e38; twelve
// FP64 operations, where pow takes more than a right-hand side). Above FLT_MAX, and at
// infinity, the estimate is zero and stays so (the caller clamps the factor from below).
SIRIUS_DEVICE __forceinline__ double inv_root5(double e) {
#ifdef __CUDA_ARCH__
    double y = double(exp2f(-0.2f * __log2f(float(e))));
#else
    double y = double(std::exp2(-0.2f * std::log2(float(e))));
#endif
    e = fmin(e, 1.7976931348623157e308);  // inf * 0 would be NaN
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int it = 0; it < 2; ++it) {
        const double y2 = mul_(y, y);
        y = fma_(mul_(0.2, y), fma_(-mul_(e, y), mul_(y2, y2), 1.0), y);
    }
    return y;
}

// The square root of a sum of squares, from rsqrt_ (2.2e-16): below 1e-280 at most 1e-140, infinity
// at infinity.
SIRIUS_DEVICE __forceinline__ double root_of_sum(double s) {
    return mul_(s, rsqrt_(fmin(fmax(s, 1e-280), 1.7976931348623157e308)));
}

}  // namespace sirius
