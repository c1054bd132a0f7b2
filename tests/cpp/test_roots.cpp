// The scalar roots of csrc/roots.cuh as host code, against bisection or powers in extended precision. Prints a line for
// what fails; the exit code is the number of failures.
#include <cmath>
#include <cstdio>
#include <random>

#include "roots.cuh"

using namespace sirius;

static int failures = 0;
static void check(bool ok, const char* what, double a, double b) {
    if (!ok) {
        ++failures;
        std::printf("%s: %.17g, %.17g\n", what, a, b);
    }
}

static std::mt19937_64 rng(1);
static double uniform(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }

// the zero by bisection in extended precision, and how far rounding may move it: FP64's half-ulp of each term of the
// cubic (seven operations) over the slope at the zero, and the correction's own bound
static double zero_of(double z0, double z1, double dz0, double dz1, double h, double& tol) {
    const long double m0 = (long double)h * dz0, m1 = (long double)h * dz1, d = (long double)z1 - z0;
    const long double c2 = 3 * d - 2 * m0 - m1, c3 = m0 + m1 - 2 * d;
    long double lo = 0, hi = 1;
    for (int i = 0; i < 100; ++i) {
        const long double s = (lo + hi) / 2, f = z0 + s * (m0 + s * (c2 + s * c3));
        if ((f < 0) == (z0 < 0)) lo = s;
        else hi = s;
    }
    const long double terms = fabsl(z0) + fabsl(m0) + fabsl(m1) + fabsl(d) + fabsl(c2) + fabsl(c3);
    tol = double(1e-15L + 7 * 0x1p-53L * terms / fabsl(m0 + lo * (2 * c2 + lo * 3 * c3)));
    return double(lo);
}

// end slopes between `least` and `most` of the chord's
static void crossings(double least, double most, int at_most, double mean) {
    const int n = 100000;
    double sum = 0, off = 0;
    int longest = 0;
    for (int i = 0; i < n; ++i) {
        const double sign = uniform(0, 1) < 0.5 ? 1 : -1, h = std::exp(uniform(-6, 1));
        const double z0 = sign * std::exp(uniform(-8, 1)), z1 = -sign * std::exp(uniform(-8, 1));
        const double a = (z1 - z0) / h * uniform(least, most), b = (z1 - z0) / h * uniform(least, most);
        int it = 0;
        double tol = 0;
        const double s = hermite_root(z0, z1, a, b, h, &it), e = zero_of(z0, z1, a, b, h, tol);
        off = std::fmax(off, std::fabs(s - e) / tol);
        sum += it;
        if (it > longest) longest = it;
    }
    check(off <= 1, "crossing: distance from the zero over its bound", off, least);
    check(longest <= at_most, "crossing: longest search", longest, least);
    check(sum / n <= mean, "crossing: mean search", sum / n, least);
}

static void exact_crossings() {
    // the chord's zero is the cubic's: f is zero at the first iterate, where the bracket ends there too
    for (double z : {1.0, -3.0, 0.125})
        for (double k : {1.0, 3.0, 7.0}) {
            int it = 0;
            const double z1 = -z * k, h = 0.5, dz = (z1 - z) / h, s = hermite_root(z, z1, dz, dz, h, &it);
            check(std::fabs(s - 1 / (1 + k)) <= 2e-16 && it <= 2, "straight crossing", s, it);
        }
    // a slope of zero at an end, and at the zero itself
    int it = 0;
    double s = hermite_root(-1.0, 1.0, 0.0, 0.0, 1.0, &it);
    check(std::fabs(s - 0.5) <= 2e-16 && it <= 2, "crossing between level ends", s, it);
    s = hermite_root(-1.0, 1.0, 6.0, 6.0, 1.0, &it);  // 8 (s - 1/2)^3 + ...: all slopes as the ends'
    check(s >= 0 && s <= 1 && it <= 60, "crossing with steep ends", s, it);
}

// e^(-1/5) to a few ulps (two Newton steps leave 3 d^2 of an estimate good to d = 1e-5, then rounding of five products),
// and a factor that never grows where the error is beyond FP32's range or infinite
static void fifth_root() {
    double off = 0;
    for (int i = 0; i < 200000; ++i) {
        const double e = std::exp(uniform(std::log(1e-15), std::log(1e38)));
        off = std::fmax(off, std::fabs(double(inv_root5(e) * powl((long double)e, 0.2L) - 1)));
    }
    check(off <= 3e-10 * 3e-10 + 6 * 0x1p-53, "fifth root: relative error", off, 0);
    for (double e : {1e39, 1e150, 1e300, 1.7976931348623157e308, HUGE_VAL}) {
        const double y = inv_root5(e);
        check(y >= 0 && y <= 1e-7, "fifth root of a huge error", y, e);
        check(std::fmax(0.1, std::fmin(2.0, 0.9 * y)) == 0.1, "step factor of a huge error", y, e);
    }
    check(std::isnan(inv_root5(NAN)), "fifth root of NaN", inv_root5(NAN), 0);
}

static void root_of_sums() {
    for (double s : {1e-279, 1e-30, 0.3, 2.0, 1e300, 1.7976931348623157e308})
        check(std::fabs(root_of_sum(s) / std::sqrt(s) - 1) <= 3 * 0x1p-53, "root of a sum", root_of_sum(s), s);
    check(root_of_sum(0.0) == 0 && root_of_sum(HUGE_VAL) == HUGE_VAL && std::isnan(root_of_sum(NAN)), "root of a sum",
          root_of_sum(HUGE_VAL), root_of_sum(NAN));
}

int main() {
    fifth_root();
    root_of_sums();
    crossings(0.99, 1.01, 4, 3.5);
    crossings(0.9, 1.1, 5, 4.0);
    crossings(0.3, 2.0, 8, 5.0);
    exact_crossings();
    return failures;
}
