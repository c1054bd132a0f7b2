// roots.cuh — scalar roots of the step control and of the event location, for the device
// and, in host-only translation units, as plain host code.
#pragma once

#include "dual.cuh"

namespace sirius {

// The zero in [0, 1] of the cubic Hermite interpolant of z over the accepted step
// (z0 and z1 have opposite signs): Newton from the chord's zero, kept inside the
// shrinking bracket (a step that leaves it bisects), to FP64 rounding, where bisection to
// the same width takes 60 iterations. Convergence is tested on the correction, before the
// bracket: the iterate has just become one of the bracket's ends, and a correction that
// rounds to zero would not lie inside. End slopes within 10 % of the chord's take 3.5 iterations in
// the mean and at most 4, within a factor of 2 to 3 4.4 and at most 6.
SIRIUS_HD __forceinline__ double hermite_root(double z0, double z1, double dz0, double dz1, double h,
                                              int* iterations = nullptr) {
    const double m0 = h * dz0, m1 = h * dz1, d = z1 - z0;
    const double c2 = 3.0 * d - 2.0 * m0 - m1, c3 = m0 + m1 - 2.0 * d;
    double lo = 0.0, hi = 1.0, s = -z0 / d;
    int it = 0;
#ifdef __CUDACC__
#pragma unroll 1
#endif
    while (it < 60) {
        ++it;
        const double f = z0 + s * (m0 + s * (c2 + s * c3));
        const double df = m0 + s * (2.0 * c2 + s * (3.0 * c3));
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

}  // namespace sirius
