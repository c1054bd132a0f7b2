// What the closed form of the Kerr-Schild right-hand side (ks_geom, csrc/spacetime.cuh) takes from r's equation, against the
// definitions that the general form uses (ks_pieces), as host code in extended precision: the potential H = (2 M r - Q^2) r^2
// / (r^4 + a^2 z^2), and l . k. Far out, and inside the ring of a naked singularity next to its disc, where r is held at 1e-5
// and no longer solves its equation.
//
// Bound: 64 roundings of 2^-64 of H's terms (2 M r and Q^2 may cancel) and of the sum of l . k's terms, and the same of what
// cancels in r^2 = (R^2 - a^2 + sd) / 2 where r is not held. Spins and charges whose squares are exact.
#include <cmath>
#include <cstdio>
#include <random>

namespace sirius {  // (before the templates that call them)
inline long double rcp_(long double x) { return 1.0L / x; }
inline long double rsqrt_(long double x) { return 1.0L / std::sqrt(x); }
inline long double sqrt_(long double x) { return std::sqrt(x); }
inline long double sqrtp_(long double x) { return std::sqrt(x); }
inline long double exp_(long double x) { return std::exp(x); }
inline long double tanh_(long double x) { return std::tanh(x); }
inline void sincos_(long double x, long double& s, long double& c) {
    s = std::sin(x);
    c = std::cos(x);
}
}  // namespace sirius
#include "spacetime.cuh"

using namespace sirius;
typedef long double real;

int main() {
    std::mt19937_64 rng(5);
    auto uniform = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); };
    const double metrics[][3] = {{0.25, -0.875, 1.25}, {1, 1.25, 0}, {1, 0, 1.25}, {0.5, 0.75, 0.625}, {1, 0.875, 0}, {0, 1.5, 0.75}};
    int failures = 0;
    for (auto& c : metrics)
        for (double Lambda : {0.0, 1e-3, -1e-3}) {
            sirius_metric s{};
            s.M = c[0]; s.a = c[1]; s.Q = c[2]; s.Lambda = Lambda;
            const MetricDev m = metric_dev(s);
            real worst = 0;
            int held = 0, n = 0;
            for (int i = 0; i < 20000; ++i) {
                const double a = std::fabs(s.a), ph = uniform(0, 6.283185307179586);
                double z, rho;
                if (i % 2) {  // near the disc (the origin where a = 0)
                    z = std::exp(uniform(std::log(1e-9), std::log(1e-1))) * (uniform(0, 1) < 0.5 ? 1 : -1);
                    rho = a > 0 ? a * std::sqrt(uniform(0.01, 0.99)) : std::exp(uniform(std::log(1e-8), std::log(1e-1)));
                } else {
                    z = uniform(-30, 30);
                    rho = uniform(0.1, 30);
                }
                const real x[4] = {0, rho * std::cos(ph), rho * std::sin(ph), z};
                const real p[4] = {-1, uniform(-2, 2), uniform(-2, 2), uniform(-2, 2)};
                KSGeom<real> G;
                KSPieces<real> P;
                real k[4], lk;
                ks_geom<true>(m, x[1], x[2], x[3], G);
                ks_pieces<real>(m, x[1], x[2], x[3], P);
                ks_velocity(m, G, p, k, lk);
                const real Rm2 = x[1] * x[1] + x[2] * x[2] + x[3] * x[3] - (real)m.a2;
                const real sd = std::sqrt(Rm2 * Rm2 + 4 * (real)m.a2 * x[3] * x[3]), raw = (Rm2 + sd) / 2;
                const bool is_held = !(raw > 1e-10L);
                const real bound = 64 * 0x1p-64L * (1 + (is_held ? 0 : (std::fabs(Rm2) + sd) / raw));
                const real terms[4] = {k[0], P.l1.v * k[1], P.l2.v * k[2], P.l3.v * k[3]};
                const real sum = terms[0] + terms[1] + terms[2] + terms[3];
                // (away from the disc l . k = l . p, whose terms may be the larger ones)
                const real size = std::fabs(terms[0]) + std::fabs(terms[1]) + std::fabs(terms[2]) + std::fabs(terms[3]) + 1 +
                                  std::fabs(p[1]) + std::fabs(p[2]) + std::fabs(p[3]);
                ++n;
                held += is_held;
                // H against the size of its own terms, 2 M r and Q^2, over the same denominator
                const real r = P.r, over = r * r / (r * r * r * r + (real)m.a2 * x[3] * x[3]);
                const real terms_h = (2 * (real)m.M * r + (real)m.Q2) * over;
                if (terms_h != 0) worst = std::fmax(worst, std::fabs(G.H - P.H.v) / terms_h / bound);
                const real off = std::fabs(lk - sum) / (size * (1 + terms_h));
                worst = std::fmax(worst, off / bound);
                if (!(off == off) || G.held != is_held) worst = 1e30L;
            }
            if (!(worst <= 1) || held < 1000 || n < 15000) {
                ++failures;
                std::printf("M %g a %g Q %g Lambda %g: %g of the bound, %d held of %d\n", s.M, s.a, s.Q, Lambda, double(worst), held, n);
            }
        }
    return failures;
}
