// spacetime.cuh — metric families on the device.
//
// Each family supplies, in any precision T:
//   rhs()          Hamilton's equations  dx^mu/dl = g^{mu nu} p_nu,
//                  dp_mu/dl = 1/2 d_mu g_{rs} k^r k^s  (PHGD001A.cpp:159-202),
//                  with d_mu g from register-resident dual numbers (dual.cuh);
//   ginv()         the inverse metric as a bilinear form (for the FP64
//                  constraint re-projection and the null value);
//   radial()       the radial coordinate of the family and its gradient dr;
//   metric_full()  g_{mu nu} and d_l g_{mu nu} (IMetric::evaluate, PHMT000A.h:38).
// The Kerr-Schild family never forms a 4x4 inverse: with the null covector
// l_mu = (1, (rx+ay)/(r^2+a^2), (ry-ax)/(r^2+a^2), z/r) (eta-null),
// g = eta + H l l  has  g^{-1} = eta - H l# l#  (l# = eta l), and the
// reference's "simplified" Lambda term -Lambda R^2/3 on g_tt
// (PHMT100A.h:362-369) is folded in exactly by a Sherman-Morrison update.
#pragma once

#include <type_traits>

#include "dual.cuh"
#include "../../include/sirius_cuda.h"

namespace sirius {

struct MetricDev {
    int family;
    int shape;
    double M, a, Q, Lambda;
    double a2, Q2, lam3, sqrtM;   // a^2, Q^2, Lambda/3
    int has_lambda;        // |Lambda| > 1e-15 (PHMT100A.h:365)
    double b0, Phi0, gtt_mt;  // Morris-Thorne: g_tt = -exp(2 Phi0)
    double vs, sigma, Rb, inv_2tanhsR;  // Alcubierre
    // FP32 copies for the single-precision paths (rounded once on the host)
    float fa, fa2, fM2, fQ2, flam3, fsqrtM;
};

// A launch constant in precision T: the FP32 copy for float, else the double.
template <class T>
SIRIUS_HD __forceinline__ T cst(double d, float) { return T(d); }
template <>
SIRIUS_HD __forceinline__ float cst<float>(double, float f) { return f; }

// Host: the per-metric constants the device code reads.
inline MetricDev metric_dev(const sirius_metric& s) {
    MetricDev m{};
    m.family = s.family;
    m.shape = s.shape;
    m.M = s.M; m.a = s.a; m.Q = s.Q; m.Lambda = s.Lambda;
    m.a2 = s.a * s.a; m.Q2 = s.Q * s.Q; m.lam3 = s.Lambda / 3.0; m.sqrtM = std::sqrt(s.M > 0.0 ? s.M : 0.0);
    m.has_lambda = std::fabs(s.Lambda) > 1e-15;
    m.b0 = s.b0; m.Phi0 = s.Phi0; m.gtt_mt = -std::exp(2.0 * s.Phi0);
    m.vs = s.vs; m.sigma = s.sigma; m.Rb = s.R;
    m.inv_2tanhsR = (s.sigma * s.R != 0.0) ? 1.0 / (2.0 * std::tanh(s.sigma * s.R)) : 0.0;
    m.fa = float(m.a); m.fa2 = float(m.a2); m.fM2 = float(2.0 * m.M); m.fQ2 = float(m.Q2);
    m.flam3 = float(m.lam3); m.fsqrtM = float(m.sqrtM);
    return m;
}

template <class T>
SIRIUS_HD __forceinline__ T tmax(T a, T b) { return a > b ? a : b; }
template <class T>
SIRIUS_HD __forceinline__ D1<T> tmax(D1<T> a, T b) { return a.v > b ? a : D1<T>(b); }
template <class T>
SIRIUS_HD __forceinline__ T value_of(T a) { return a; }
template <class T>
SIRIUS_HD __forceinline__ T value_of(D1<T> a) { return a.v; }

// ---------------------------------------------------------------------------
// Kerr-Schild family (PHMT100A.h:198-396): H and l_i as dual numbers.
// r solves r^4 - (R^2 - a^2) r^2 - a^2 z^2 = 0; its gradient enters as the
// implicit-function seed  dr = (r x, r y, z (r^2 + a^2) / r) / sqrt(disc).
// ---------------------------------------------------------------------------
template <class T>
struct KSPieces {
    D3<T> H, l1, l2, l3;
    T r;
};

template <class T>
SIRIUS_HD __forceinline__ void ks_pieces(const MetricDev& m, T x, T y, T z, KSPieces<T>& o) {
    const T a = T(m.a), a2 = T(m.a2);
    const T R2 = x * x + y * y + z * z;
    const T Rm2 = R2 - a2;
    const T disc = tmax(Rm2 * Rm2 + T(4) * a2 * z * z, T(1e-20));
    const T sd = sqrtp_(disc);
    const T r2 = tmax((Rm2 + sd) * T(0.5), T(1e-10));
    const T r = sqrtp_(r2);
    const T isd = rcp_(sd);
    const T ir = rcp_(r);
    const D3<T> rd = dwith(r, r * x * isd, r * y * isd, z * (r2 + a2) * isd * ir);
    const D3<T> X = dvar(x, 0), Y = dvar(y, 1), Z = dvar(z, 2);
    const D3<T> rr2 = rd * rd;
    const D3<T> iden = inv(rr2 + a2);
    o.l1 = (rd * X + Y * a) * iden;
    o.l2 = (rd * Y - X * a) * iden;
    o.l3 = Z * dwith(ir, -ir * ir * rd.d[0], -ir * ir * rd.d[1], -ir * ir * rd.d[2]);
    const D3<T> num = (rd * T(2.0 * m.M) - T(m.Q2)) * rr2;
    const D3<T> fden = rr2 * rr2 + Z * Z * a2;
    o.H = num * inv(fden);
    o.r = r;
}

// The Kerr-Schild right-hand side k = g^{-1} p, f = dp / dlambda with the forward-mode
// tangents of ks_pieces propagated term by term: the coordinate seeds dx = (1, 0, 0), ... have
// zero components, and an IEEE product with a zero cannot be dropped at compile time
// (inf * 0 is NaN), so the generic dual arithmetic pays for every one of them.
// Here only the non-zero terms are formed:
//   dr  = (r x, r y, z (r^2 + a^2) / r) / sqrt(disc)
//   d(1/(r^2 + a^2)) = -2 r / (r^2 + a^2)^2 dr
//   d l1 = (x dr + (r, a, 0)) / (r^2 + a^2) + (r x + a y) d(1/(r^2 + a^2)), l2 alike
//   d l3 = (0, 0, 1) / r - z / r^2 dr
//   d H  = ((2 M r^2 + 2 r (2 M r - Q^2) - H 4 r^3) dr - H (0, 0, 2 a^2 z)) / fden
// with num = (2 M r - Q^2) r^2, fden = r^4 + a^2 z^2, H = num / fden.
template <class T>
SIRIUS_HD __forceinline__ void ks_rhs_terms(const MetricDev& m, const T x[4], const T p[4], T k[4], T f[4]) {
    const T a = cst<T>(m.a, m.fa), a2 = cst<T>(m.a2, m.fa2);
    const T X = x[1], Y = x[2], Z = x[3];
    const T zz = Z * Z;
    const T R2 = X * X + Y * Y + zz;
    const T Rm2 = R2 - a2;
    const T a2zz = a2 * zz;
    const T disc = tmax(Rm2 * Rm2 + T(4) * a2zz, T(1e-20));
    const T sd = sqrtp_(disc);
    const T r2 = tmax((Rm2 + sd) * T(0.5), T(1e-10));
    const T r = sqrtp_(r2);
    const T isd = rcp_(sd), ir = rcp_(r);
    const T den = r2 + a2;
    const T risd = r * isd;
    const T rx = risd * X, ry = risd * Y, rz = Z * den * isd * ir;
    const T iden = rcp_(den);
    const T gi = -T(2) * r * iden * iden;
    const T n1 = r * X + a * Y, n2 = r * Y - a * X;
    const T l1 = n1 * iden, l2 = n2 * iden;
    const T n1g = n1 * gi, n2g = n2 * gi;
    const T l1d0 = (X * rx + r) * iden + n1g * rx, l1d1 = (X * ry + a) * iden + n1g * ry,
            l1d2 = X * rz * iden + n1g * rz;
    const T l2d0 = (Y * rx - a) * iden + n2g * rx, l2d1 = (Y * ry + r) * iden + n2g * ry,
            l2d2 = Y * rz * iden + n2g * rz;
    const T l3 = Z * ir;
    const T zi2 = -l3 * ir;
    const T l3d0 = zi2 * rx, l3d1 = zi2 * ry, l3d2 = zi2 * rz + ir;
    const T M2 = cst<T>(2.0 * m.M, m.fM2);
    const T q = M2 * r - cst<T>(m.Q2, m.fQ2);
    const T fden = r2 * r2 + a2zz;
    const T ifd = rcp_(fden);
    const T H = q * r2 * ifd;
    const T w = (M2 * r2 + T(2) * r * q - H * T(4) * r2 * r) * ifd;
    const T Hd0 = w * rx, Hd1 = w * ry, Hd2 = w * rz - H * ifd * T(2) * a2 * Z;
    // k = g^{-1} p = eta p - H l# (l# . p), l# = (-1, l1, l2, l3)
    const T lp = -p[0] + l1 * p[1] + l2 * p[2] + l3 * p[3];
    const T Hlp = H * lp;
    k[0] = -p[0] + Hlp;
    k[1] = p[1] - l1 * Hlp;
    k[2] = p[2] - l2 * Hlp;
    k[3] = p[3] - l3 * Hlp;
    if (m.has_lambda) {
        const T c = cst<T>(m.lam3, m.flam3) * R2;
        const T w0 = -T(1) - H, w1 = H * l1, w2 = H * l2, w3 = H * l3;
        const T s = c * (w0 * p[0] + w1 * p[1] + w2 * p[2] + w3 * p[3]) * rcp_(T(1) + c * (T(1) + H));
        k[0] += s * w0; k[1] += s * w1; k[2] += s * w2; k[3] += s * w3;
    }
    // dp_lambda = 1/2 dH (l.k)^2 + H (l.k)(dl.k) [- Lambda x_lambda (k^0)^2 / 3]
    const T lk = k[0] + l1 * k[1] + l2 * k[2] + l3 * k[3];
    const T hlk = T(0.5) * lk;
    f[0] = T(0);
    f[1] = lk * (Hd0 * hlk + H * (l1d0 * k[1] + l2d0 * k[2] + l3d0 * k[3]));
    f[2] = lk * (Hd1 * hlk + H * (l1d1 * k[1] + l2d1 * k[2] + l3d1 * k[3]));
    f[3] = lk * (Hd2 * hlk + H * (l1d2 * k[1] + l2d2 * k[2] + l3d2 * k[3]));
    if (m.has_lambda) {
        const T qq = cst<T>(m.lam3, m.flam3) * k[0] * k[0];
        f[1] -= qq * X; f[2] -= qq * Y; f[3] -= qq * Z;
    }
}

// The same right-hand side in closed form, the one the FP64 arithmetic runs. With
// sd = sqrt((R^2 - a^2)^2 + 4 a^2 z^2) the implicit equation of r gives
// r^4 + a^2 z^2 = r^2 sd, so H = (2 M r - Q^2) / sd, and with dr = (r x, r y,
// z (r^2 + a^2) / r) / sd every gradient is a multiple of dr plus an explicit term.
// The sum over l's components is formed before the gradient's, so that
//   d_i l_j k^j = S dr_i + E_i,
//     S = (k^x x + k^y y - 2 r (l_x k^x + l_y k^y)) / (r^2 + a^2) - k^z z / r^2,
//     E = ((r k^x - a k^y) / (r^2 + a^2), (a k^x + r k^y) / (r^2 + a^2), k^z / r),
//   d_i H = w dr_i - 2 H a^2 z / (r^2 sd) delta_iz,  w = (2 M + 2 (2 M r - Q^2) / r - 4 H r) / sd,
//   dp_i = (l.k) ((w (l.k) / 2 + H S) dr_i + H E_i - H a^2 z (l.k) / (r^2 sd) delta_iz).
// l is null for eta, so l.k = l#.p where k = g^{-1} p carries no Lambda term.
// The FP64 kernels are bound by the issue and latency of their FP64 instructions,
// and an FP64 root or reciprocal is a sequence of about ten: this form takes two
// reciprocal square roots and one reciprocal where the terms take two square
// roots and four reciprocals, and 94 operations instead of 143 (717 x 405 FP64
// frame 8.73 -> 7.45 ms from this alone). The FP32 stages of the mixed DP45 path keep the terms:
// the two forms round differently, near the critical curve FP32 roundings reach the image, and which
// of the two images is nearer to FP64 has not been measured.
// In three parts: what depends on the position alone (KSGeom), the velocity and the
// force at a momentum, so that the symplectic integrator, which takes two kicks and
// a drift at each position, evaluates the geometry once.
//
// All of it rests on r solving its equation. Where r is held at 1e-5 (inside the ring, next
// to its disc) r^2 sd is not r^4 + a^2 z^2 and l is not null: there 1 / sd gives way to
// r^2 / (r^4 + a^2 z^2) wherever it stands for that, and l.k is formed from k, which makes this
// the terms' right-hand side again. RING compiles that in; only rays that no horizon stops
// need it (FrameDev::cls). It cost the others 6 % in FP64 and 3 % in symplectic steps.
template <class T>
struct KSGeom {
    T X, Y, Z, r, ir, isd, iden, den, l1, l2, l3, H, w, c, hz;  // c = Lambda R^2 / 3, hz = a^2 z / (r sd)
    bool held;  // r is the least one
};

template <bool RING, class T>
SIRIUS_HD __forceinline__ void ks_geom(const MetricDev& m, T X, T Y, T Z, KSGeom<T>& G) {
    using C = typename scalar_of<T>::type;
    const C a = cst<C>(m.a, m.fa), a2 = cst<C>(m.a2, m.fa2), M2 = cst<C>(2.0 * m.M, m.fM2);
    const T zz = mul_(Z, Z);
    const T R2 = fma_(X, X, fma_(Y, Y, zz));
    const T Rm2 = R2 - a2;
    const T a2zz = mul_(a2, zz);
    const T disc = tmax(fma_(Rm2, Rm2, mul_(C(4), a2zz)), C(1e-20));
    const T isd = rsqrt_(disc);
    const T r2 = tmax(mul_(fma_(disc, isd, Rm2), C(0.5)), C(1e-10));
    const T ir = rsqrt_(r2);
    const T r = mul_(r2, ir);
    const T den = r2 + a2;
    const T iden = rcp_(den);
    T ih = isd;  // r^2 / (r^4 + a^2 z^2)
    G.held = RING && !(value_of(r2) > C(1e-10));
    if (G.held) ih = mul_(r2, rcp_(fma_(r2, r2, a2zz)));
    const T q = fma_(M2, r, -cst<C>(m.Q2, m.fQ2));
    G.X = X; G.Y = Y; G.Z = Z; G.r = r; G.ir = ir; G.isd = isd; G.iden = iden; G.den = den;
    G.l1 = mul_(fma_(r, X, mul_(a, Y)), iden);
    G.l2 = mul_(fma_(r, Y, mul_(-a, X)), iden);
    G.l3 = mul_(Z, ir);
    G.H = mul_(q, ih);
    G.w = mul_(fma_(mul_(C(2), q), ir, fma_(mul_(C(-4), G.H), r, M2)), ih);
    G.hz = mul_(mul_(a2, G.l3), ih);
    G.c = T(0);
    if (m.has_lambda) G.c = mul_(cst<C>(m.lam3, m.flam3), R2);
}

// k = g^{-1} p = eta p - H l# (l# . p), l# = (-1, l1, l2, l3); lk = l . k
template <class T>
SIRIUS_HD __forceinline__ void ks_velocity(const MetricDev& m, const KSGeom<T>& G, const T p[4], T k[4], T& lk) {
    using C = typename scalar_of<T>::type;
    const T lp = fma_(G.l3, p[3], fma_(G.l2, p[2], fma_(G.l1, p[1], -p[0])));
    const T Hlp = mul_(G.H, lp);
    k[0] = Hlp - p[0];
    k[1] = fma_(-G.l1, Hlp, p[1]);
    k[2] = fma_(-G.l2, Hlp, p[2]);
    k[3] = fma_(-G.l3, Hlp, p[3]);
    lk = lp;
    if (m.has_lambda) {
        const T w0 = -C(1) - G.H, w1 = mul_(G.H, G.l1), w2 = mul_(G.H, G.l2), w3 = mul_(G.H, G.l3);
        const T wp = fma_(w3, p[3], fma_(w2, p[2], fma_(w1, p[1], mul_(w0, p[0]))));
        const T s = mul_(mul_(G.c, wp), rcp_(fma_(G.c, C(1) + G.H, C(1))));
        k[0] = fma_(s, w0, k[0]); k[1] = fma_(s, w1, k[1]); k[2] = fma_(s, w2, k[2]); k[3] = fma_(s, w3, k[3]);
    }
    if (m.has_lambda || G.held) lk = fma_(G.l3, k[3], fma_(G.l2, k[2], fma_(G.l1, k[1], k[0])));
}

// f_i = dp_i / dl, i = 1..3 (f_0 = 0: the metric is static), from the velocity
template <class T>
SIRIUS_HD __forceinline__ void ks_force(const MetricDev& m, const KSGeom<T>& G, const T k[4], T lk, T f[4]) {
    using C = typename scalar_of<T>::type;
    const C a = cst<C>(m.a, m.fa);
    const T xk = fma_(G.X, k[1], mul_(G.Y, k[2])), l12 = fma_(G.l1, k[1], mul_(G.l2, k[2]));
    const T S = fma_(fma_(mul_(C(-2), G.r), l12, xk), G.iden, mul_(mul_(-k[3], G.l3), G.ir));
    const T Hlk = mul_(G.H, lk), e = mul_(Hlk, G.iden);
    const T g = mul_(mul_(lk, fma_(mul_(C(0.5), G.w), lk, mul_(G.H, S))), G.isd);
    const T gr = mul_(g, G.r);
    f[0] = T(0);
    f[1] = fma_(gr, G.X, mul_(e, fma_(G.r, k[1], mul_(-a, k[2]))));
    f[2] = fma_(gr, G.Y, mul_(e, fma_(a, k[1], mul_(G.r, k[2]))));
    f[3] = mul_(G.ir, fma_(mul_(g, G.den), G.Z, mul_(Hlk, fma_(-G.hz, lk, k[3]))));
    if (m.has_lambda) {  // - Lambda x_i (k^0)^2 / 3
        const T qq = mul_(cst<C>(m.lam3, m.flam3), mul_(k[0], k[0]));
        f[1] = fma_(-qq, G.X, f[1]); f[2] = fma_(-qq, G.Y, f[2]); f[3] = fma_(-qq, G.Z, f[3]);
    }
}

template <bool RING, class T>
SIRIUS_HD __forceinline__ void ks_rhs_closed(const MetricDev& m, const T x[4], const T p[4], T k[4], T f[4]) {
    KSGeom<T> G;
    T lk;
    ks_geom<RING>(m, x[1], x[2], x[3], G);
    ks_velocity(m, G, p, k, lk);
    ks_force(m, G, k, lk, f);
}

// The Kerr-Schild right-hand side of precision T: the closed form in FP64, the
// terms otherwise (and for the operation count, which is the FP32 kernel's).
template <bool RING, class T>
SIRIUS_HD __forceinline__ void ks_rhs_fast(const MetricDev& m, const T x[4], const T p[4], T k[4], T f[4]) {
    if constexpr (std::is_same<T, double>::value) ks_rhs_closed<RING>(m, x, p, k, f);
    else ks_rhs_terms(m, x, p, k, f);
}

// ---------------------------------------------------------------------------
// Morris-Thorne (PHMT101A.h:195-345), chart (t, r, theta, phi); r clamped to
// >= 1.001 b0 as the reference does (:293); g diagonal.
// ---------------------------------------------------------------------------
template <class T>
SIRIUS_HD __forceinline__ D3<T> mt_grr(const MetricDev& m, T r) {
    const T b0 = T(m.b0);
    const D3<T> R = dvar(tmax(r, b0 * T(1.001)), 0);
    D3<T> b;
    if (m.shape == SIRIUS_WORMHOLE_ZERO_TIDAL) b = dconst(b0);
    else if (m.shape == SIRIUS_WORMHOLE_ABSURDLY_BENIGN) b = (dconst(T(2)) - inv(R) * b0) * b0;
    else b = inv(R) * (b0 * b0);  // Ellis
    D3<T> f = dconst(T(1)) - b * inv(R);
    if (f.v < T(1e-10)) f = dconst(T(1e-10));
    return inv(f);
}

template <class T>
SIRIUS_HD __forceinline__ void mt_rhs(const MetricDev& m, const T x[4], const T p[4], T k[4], T f[4]) {
    const T r = tmax(x[1], T(m.b0) * T(1.001));
    T s, c;
    sincos_(x[2], s, c);
    const T s2 = tmax(s * s, T(1e-24));
    const D3<T> grr = mt_grr(m, x[1]);
    const T r2 = r * r;
    k[0] = p[0] * rcp_(T(m.gtt_mt));
    k[1] = p[1] * rcp_(grr.v);
    k[2] = p[2] * rcp_(r2);
    k[3] = p[3] * rcp_(r2 * s2);
    f[0] = T(0);
    f[1] = T(0.5) * grr.d[0] * k[1] * k[1] + r * (k[2] * k[2] + s2 * k[3] * k[3]);
    f[2] = r2 * s * c * k[3] * k[3];
    f[3] = T(0);
}

// ---------------------------------------------------------------------------
// Alcubierre (PHMT102A.h:136-229), Cartesian, static bubble at the origin:
// g_tt = -(1 - v^2 f^2), g_tx = -v f;  g^{tt} = -1, g^{tx} = -v f, g^{xx} = 1 - v^2 f^2.
// ---------------------------------------------------------------------------
template <class T>
SIRIUS_HD __forceinline__ D3<T> alc_f(const MetricDev& m, T x, T y, T z) {
    const T rs = tmax(sqrt_(x * x + y * y + z * z), T(1e-10));
    const T irs = rcp_(rs);
    const D3<T> R = dwith(rs, x * irs, y * irs, z * irs);
    const T sg = T(m.sigma), Rb = T(m.Rb);
    // outside the bubble's wall both tanh are exactly 1, and f and its gradient exactly
    // 0: nearly all of a ray's path, without its two tanh (12 frames of four families,
    // 64^2 to 320^2: 10.12 -> 9.67 ms with the reciprocals of the other forms)
    if (tanh_is_one((rs - Rb) * sg) && tanh_is_one((rs + Rb) * sg)) return dconst(T(0));
    return (dtanh((R + Rb) * sg) - dtanh((R - Rb) * sg)) * T(m.inv_2tanhsR);
}

template <class T>
SIRIUS_HD __forceinline__ void alc_rhs(const MetricDev& m, const T x[4], const T p[4], T k[4], T f[4]) {
    const D3<T> F = alc_f(m, x[1], x[2], x[3]);
    const T v = T(m.vs), vf = v * F.v;
    k[0] = -p[0] - vf * p[1];
    k[1] = -vf * p[0] + (T(1) - vf * vf) * p[1];
    k[2] = p[2];
    k[3] = p[3];
    // dp = v df (v f (k^t)^2 - k^t k^x)
    const T q = v * (vf * k[0] * k[0] - k[0] * k[1]);
    f[0] = T(0);
    f[1] = q * F.d[0];
    f[2] = q * F.d[1];
    f[3] = q * F.d[2];
}

// FAM selects the metric family at compile time (a kernel specialised for one
// family carries one right-hand side); kAnyFamily dispatches on m.family.
constexpr int kAnyFamily = -1;
// Kerr-Schild frames whose rays may come to where r is held (KSGeom): no horizon stops them before.
// They have kernels of their own, without one-frame forms (charged, Q = 1.3, 512^2: FP64 2.9 ms, 2.5
// without the test for held r and 6.0 with the general forms throughout).
constexpr int kClassRing = 3;
// Whether a kernel of family FAM carries the forms of that region.
template <int FAM>
constexpr bool kRing = FAM == kAnyFamily || FAM == kClassRing;

template <class T, int FAM = kAnyFamily>
SIRIUS_HD __forceinline__ void rhs(const MetricDev& m, const T x[4], const T p[4], T k[4], T f[4]) {
    if constexpr (FAM == SIRIUS_METRIC_KERR_SCHILD) ks_rhs_fast<false>(m, x, p, k, f);
    else if constexpr (FAM == kClassRing) ks_rhs_fast<true>(m, x, p, k, f);
    else if constexpr (FAM == SIRIUS_METRIC_MORRIS_THORNE) mt_rhs(m, x, p, k, f);
    else if constexpr (FAM == SIRIUS_METRIC_ALCUBIERRE) alc_rhs(m, x, p, k, f);
    else if (m.family == SIRIUS_METRIC_KERR_SCHILD) ks_rhs_fast<true>(m, x, p, k, f);
    else if (m.family == SIRIUS_METRIC_MORRIS_THORNE) mt_rhs(m, x, p, k, f);
    else alc_rhs(m, x, p, k, f);
}

// Whether a ray of family FAM (or, for kAnyFamily, of m.family) is of family F.
template <int FAM>
SIRIUS_HD __forceinline__ bool is_family(const MetricDev& m, int F) {
    if constexpr (FAM == kAnyFamily) return m.family == F;
    else if constexpr (FAM == kClassRing) return F == SIRIUS_METRIC_KERR_SCHILD;
    else return FAM == F;
}

// ---------------------------------------------------------------------------
// Inverse metric as a bilinear form, evaluated once at x for up to three
// covectors: out = {g^{-1}(u,u), g^{-1}(u,v), g^{-1}(v,v)}. Also returns the
// family's radial coordinate r and its gradient d (the projection direction).
// ---------------------------------------------------------------------------
struct InvForm {
    double r;      // radial coordinate (KS: Boyer-Lindquist r; MT: r; Alcubierre: R)
    double d[4];   // dr
    double H, l[4], c, w[4], sm;  // KS pieces
    double diag[4];               // MT
    double vf;                    // Alcubierre
};

template <bool RING = true>
__device__ __forceinline__ void inv_form(const MetricDev& m, const double x[4], InvForm& F) {
    F.d[0] = 0.0;
    if (m.family == SIRIUS_METRIC_MORRIS_THORNE) {
        const double r = fmax(x[1], m.b0 * 1.001);
        const double s = sin(x[2]);
        const double s2 = fmax(s * s, 1e-24);
        const D3<double> grr = mt_grr<double>(m, x[1]);
        F.r = x[1];
        F.d[1] = 1.0; F.d[2] = 0.0; F.d[3] = 0.0;
        const double ir2 = rcp_(mul_(r, r));
        F.diag[0] = rcp_(m.gtt_mt); F.diag[1] = rcp_(grr.v); F.diag[2] = ir2; F.diag[3] = mul_(ir2, rcp_(s2));
        return;
    }
    const double X = x[1], Y = x[2], Z = x[3];
    const double zz = mul_(Z, Z), R2 = fma_(X, X, fma_(Y, Y, zz));
    if (m.family == SIRIUS_METRIC_ALCUBIERRE) {
        const double iR = rsqrt_(fmax(R2, 1e-300)), Rr = mul_(R2, iR);  // (the bubble's centre: r = 0, no direction)
        F.r = Rr;
        F.d[1] = mul_(X, iR); F.d[2] = mul_(Y, iR); F.d[3] = mul_(Z, iR);
        const D3<double> f = alc_f<double>(m, X, Y, Z);
        F.vf = mul_(m.vs, f.v);
        return;
    }
    // (roots and reciprocals as in ks_rhs_closed: H = (2 M r - Q^2) / sd)
    const double a2 = m.a2, Rm2 = R2 - a2, a2zz = mul_(a2, zz);
    const double disc = fmax(fma_(Rm2, Rm2, mul_(4.0, a2zz)), 1e-20);
    const double isd = rsqrt_(disc);
    const double r2 = fmax(mul_(0.5, fma_(disc, isd, Rm2)), 1e-10);
    const double ir = rsqrt_(r2), r = mul_(r2, ir);
    const double den = r2 + a2, iden = rcp_(den);
    const double q = fma_(2.0 * m.M, r, -m.Q2);
    F.r = r;
    F.d[1] = mul_(mul_(r, X), isd); F.d[2] = mul_(mul_(r, Y), isd); F.d[3] = mul_(mul_(Z, den), mul_(ir, isd));
    F.l[0] = -1.0;  // l# = eta l
    F.l[1] = mul_(fma_(r, X, mul_(m.a, Y)), iden);
    F.l[2] = mul_(fma_(r, Y, mul_(-m.a, X)), iden);
    F.l[3] = mul_(Z, ir);
    F.H = mul_(q, isd);
    if (RING && !(r2 > 1e-10)) {  // r is held (KSGeom): H as in the terms, and for a = 0 the radial direction
        F.H = mul_(mul_(q, r2), rcp_(fma_(r2, r2, a2zz)));
        if (m.a == 0.0) {
            const double iR = rsqrt_(fmax(R2, 1e-300));
            F.d[1] = mul_(X, iR); F.d[2] = mul_(Y, iR); F.d[3] = mul_(Z, iR);
        }
    }
    F.w[0] = -1.0 - F.H; F.w[1] = mul_(F.H, F.l[1]); F.w[2] = mul_(F.H, F.l[2]); F.w[3] = mul_(F.H, F.l[3]);
    F.c = 0.0;
    F.sm = 0.0;
    if (m.has_lambda) {
        F.c = mul_(m.lam3, R2);
        F.sm = F.c / fma_(F.c, 1.0 + F.H, 1.0);
    }
}

__device__ __forceinline__ double inv_apply(const MetricDev& m, const InvForm& F, const double u[4], const double v[4]) {
    if (m.family == SIRIUS_METRIC_MORRIS_THORNE)
        return fma_(mul_(F.diag[3], u[3]), v[3],
                    fma_(mul_(F.diag[2], u[2]), v[2], fma_(mul_(F.diag[1], u[1]), v[1], mul_(mul_(F.diag[0], u[0]), v[0]))));
    if (m.family == SIRIUS_METRIC_ALCUBIERRE) {
        const double cross = fma_(u[0], v[1], mul_(u[1], v[0])), g11 = fma_(-F.vf, F.vf, 1.0);
        return fma_(u[3], v[3], fma_(u[2], v[2], fma_(mul_(g11, u[1]), v[1], fma_(-F.vf, cross, mul_(-u[0], v[0])))));
    }
    const double eta = fma_(u[3], v[3], fma_(u[2], v[2], fma_(u[1], v[1], mul_(-u[0], v[0]))));
    const double lu = fma_(F.l[3], u[3], fma_(F.l[2], u[2], fma_(F.l[1], u[1], mul_(F.l[0], u[0]))));
    const double lv = fma_(F.l[3], v[3], fma_(F.l[2], v[2], fma_(F.l[1], v[1], mul_(F.l[0], v[0]))));
    double s = fma_(mul_(-F.H, lu), lv, eta);
    if (m.has_lambda) {
        const double wu = fma_(F.w[3], u[3], fma_(F.w[2], u[2], fma_(F.w[1], u[1], mul_(F.w[0], u[0]))));
        const double wv = fma_(F.w[3], v[3], fma_(F.w[2], v[2], fma_(F.w[1], v[1], mul_(F.w[0], v[0]))));
        s = fma_(mul_(F.sm, wu), wv, s);
    }
    return s;
}

// E/L_z/Carter-preserving constraint re-projection: p <- p + alpha dr with the
// root alpha of g^{-1}(p + a dr, p + a dr) = 0 of smallest magnitude — the
// chart-independent form of SymplecticIntegratorD::renormalizeNull's p_r
// solve (PHSI001A.h:366-418). Returns the null value before projection.
__device__ __forceinline__ double project_null(const MetricDev& m, const InvForm& F, double p[4]) {
    const double A = inv_apply(m, F, F.d, F.d);
    const double B = 2.0 * inv_apply(m, F, p, F.d);
    const double C = inv_apply(m, F, p, p);
    const double disc = fma_(B, B, mul_(mul_(-4.0, A), C));
    if (disc < 0.0 || fabs(A) < 1e-15) return C;
    const double sq = mul_(disc, rsqrt_(fmax(disc, 1e-280)));
    const double q = mul_(-0.5, B + (B >= 0.0 ? sq : -sq));
    if (q == 0.0) return C;
    const double alpha = mul_(C, rcp_(q));
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = fma_(alpha, F.d[i], p[i]);
    return C;
}

// The same re-projection for the Kerr-Schild family without Lambda, where the
// coefficients are short: l is tangent to the null congruence on which r is an affine
// parameter, so l . dr = 1, and |dr|^2 = (r^2 + a^2) / sd, which leaves
//   A = g^{-1}(dr, dr) = (r^2 + a^2) / sd - H,   B / 2 = g^{-1}(p, dr) = p . dr - H l#.p.
// Only the null value C = g^{-1}(p, p) always needs FP64: it is a difference of O(p^2)
// terms that must survive to ~1e-16 of them. The mixed path (T = float) takes the
// direction dr and the coefficients in FP32: they only set alpha = C / q, which needs
// single-precision relative accuracy there, and the constraint left after the update is
// ~1e-7 C; the FP64 path (T = double) keeps everything in FP64. Returns C; r_out = r;
// moved: the update is beyond what the stored f(x, p) resolves (1e-6 of p with FP32
// storage, 1e-10 in FP64).
template <class T, bool RING>
__device__ __forceinline__ double project_null_ks(const MetricDev& m, const double x[4], double p[4], double& r_out,
                                                  bool& moved) {
    moved = false;
    const double X = x[1], Y = x[2], Z = x[3];
    const double a = m.a, a2 = m.a2;
    const double zz = mul_(Z, Z), R2 = fma_(X, X, fma_(Y, Y, zz)), Rm2 = R2 - a2, a2zz = mul_(a2, zz);
    const double disc2 = fmax(fma_(Rm2, Rm2, mul_(4.0, a2zz)), 1e-20);
    const double isd = rsqrt_(disc2);
    const double r2 = fmax(mul_(0.5, fma_(disc2, isd, Rm2)), 1e-10);
    const double ir = rsqrt_(r2), r = mul_(r2, ir);
    r_out = r;
    const double den = r2 + a2, iden = rcp_(den);
    const double l1 = mul_(fma_(r, X, mul_(a, Y)), iden), l2 = mul_(fma_(r, Y, mul_(-a, X)), iden), l3 = mul_(Z, ir);
    const bool held = RING && !(r2 > 1e-10);  // r does not solve its equation there (KSGeom)
    const double q2 = fma_(2.0 * m.M, r, -m.Q2);
    double H = mul_(q2, isd);
    if (held) H = mul_(mul_(q2, r2), rcp_(fma_(r2, r2, a2zz)));
    const double lp = fma_(l3, p[3], fma_(l2, p[2], fma_(l1, p[1], -p[0])));
    const double pp = fma_(p[3], p[3], fma_(p[2], p[2], fma_(p[1], p[1], mul_(-p[0], p[0]))));
    const double C = fma_(mul_(-H, lp), lp, pp);
    const T isdt = T(isd), rs = mul_(T(r), isdt), dt = mul_(T(den), isdt);
    T d1 = mul_(rs, T(X)), d2 = mul_(rs, T(Y)), d3 = mul_(mul_(T(Z), dt), T(ir));
    T ld = T(1), dd = dt;  // l . dr, |dr|^2
    if (held) {
        if (sizeof(T) == sizeof(double) && m.a == 0.0) {
            const double iR = rsqrt_(fmax(R2, 1e-300));
            d1 = T(mul_(X, iR)); d2 = T(mul_(Y, iR)); d3 = T(mul_(Z, iR));
        }
        ld = fma_(T(l3), d3, fma_(T(l2), d2, mul_(T(l1), d1)));
        dd = fma_(d3, d3, fma_(d2, d2, mul_(d1, d1)));
    }
    const T p1 = T(p[1]), p2 = T(p[2]), p3 = T(p[3]);
    const T Ht = mul_(T(H), ld);
    const T A = fma_(-Ht, ld, dd);
    const T pd = fma_(p3, d3, fma_(p2, d2, mul_(p1, d1)));
    const T B = mul_(T(2), fma_(-Ht, T(lp), pd));
    const T Ct = T(C);
    const T disc = fma_(B, B, mul_(mul_(T(-4), A), Ct));
    // (at the horizon A = 0, exactly so in FP32 for some rays: C / q needs no division by A)
    if (!(disc >= T(0)) || (sizeof(T) == sizeof(double) && fabs(A) < T(1e-15))) return C;
    T sq;
    if constexpr (sizeof(T) == sizeof(double)) sq = mul_(disc, rsqrt_(fmax(disc, 1e-280)));
    else sq = sqrtf(disc);
    const T q = mul_(T(-0.5), B + (B >= T(0) ? sq : -sq));
    if (q == T(0)) return C;
    const T al = mul_(Ct, rcp_(q));
    const double alpha = double(al);
    p[1] = fma_(alpha, double(d1), p[1]);
    p[2] = fma_(alpha, double(d2), p[2]);
    p[3] = fma_(alpha, double(d3), p[3]);
    const float pm = fmaxf(fmaxf(fabsf(float(p[0])), fabsf(float(p1))), fmaxf(fabsf(float(p2)), fabsf(float(p3))));
    const float dm = fmaxf(fmaxf(fabsf(float(d1)), fabsf(float(d2))), fabsf(float(d3)));
    moved = fabsf(float(al)) * dm > (sizeof(T) == sizeof(double) ? 1e-10f : 1e-6f) * pm;
    return C;
}

// ---------------------------------------------------------------------------
// The metric alone, FP64, closed form (no derivatives): g[16].
// ---------------------------------------------------------------------------
__device__ __forceinline__ void metric_g(const MetricDev& m, const double x[4], double g[16]) {
    for (int i = 0; i < 16; ++i) g[i] = 0.0;
    if (m.family == SIRIUS_METRIC_MORRIS_THORNE) {
        const double r = fmax(x[1], m.b0 * 1.001);
        const double s = sin(x[2]);
        g[0] = m.gtt_mt;
        g[5] = mt_grr<double>(m, x[1]).v;
        g[10] = r * r;
        g[15] = r * r * s * s;
        return;
    }
    if (m.family == SIRIUS_METRIC_ALCUBIERRE) {
        const double vf = m.vs * alc_f<double>(m, x[1], x[2], x[3]).v;
        g[0] = -(1.0 - vf * vf);
        g[1] = g[4] = -vf;
        g[5] = g[10] = g[15] = 1.0;
        return;
    }
    InvForm F;
    inv_form(m, x, F);
    const double l[4] = {1.0, F.l[1], F.l[2], F.l[3]};  // covariant l
    for (int a = 0; a < 4; ++a)
        for (int b = 0; b < 4; ++b) g[4 * a + b] = ((a == b) ? (a == 0 ? -1.0 : 1.0) : 0.0) + F.H * l[a] * l[b];
    if (m.has_lambda) g[0] -= m.lam3 * (x[1] * x[1] + x[2] * x[2] + x[3] * x[3]);
}

// ---------------------------------------------------------------------------
// Full metric and derivatives (IMetric::evaluate): g[16], dg[64], dg[l*16+m*4+n].
// ---------------------------------------------------------------------------
template <class T>
__device__ void metric_full(const MetricDev& m, const T x[4], T g[16], T dg[64]) {
    for (int i = 0; i < 16; ++i) g[i] = T(0);
    for (int i = 0; i < 64; ++i) dg[i] = T(0);
    if (m.family == SIRIUS_METRIC_KERR_SCHILD) {
        KSPieces<T> P;
        ks_pieces(m, x[1], x[2], x[3], P);
        const D3<T> one = dconst(T(1));
        const D3<T> l[4] = {one, P.l1, P.l2, P.l3};
        for (int a = 0; a < 4; ++a)
            for (int b = 0; b < 4; ++b) {
                const D3<T> h = P.H * l[a] * l[b];
                const T eta = (a == b) ? (a == 0 ? T(-1) : T(1)) : T(0);
                g[4 * a + b] = eta + h.v;
                for (int q = 0; q < 3; ++q) dg[16 * (q + 1) + 4 * a + b] = h.d[q];
            }
        if (m.has_lambda) {
            g[0] -= T(m.lam3) * (x[1] * x[1] + x[2] * x[2] + x[3] * x[3]);
            for (int q = 0; q < 3; ++q) dg[16 * (q + 1)] -= T(2) * T(m.lam3) * x[q + 1];
        }
    } else if (m.family == SIRIUS_METRIC_MORRIS_THORNE) {
        const T r = tmax(x[1], T(m.b0) * T(1.001));
        const T s = sin(x[2]), c = cos(x[2]);
        const D3<T> grr = mt_grr(m, x[1]);
        g[0] = T(m.gtt_mt);
        g[5] = grr.v;
        g[10] = r * r;
        g[15] = r * r * s * s;
        dg[16 + 5] = grr.d[0];
        dg[16 + 10] = T(2) * r;
        dg[16 + 15] = T(2) * r * s * s;
        dg[32 + 15] = T(2) * r * r * s * c;
    } else {
        const D3<T> F = alc_f(m, x[1], x[2], x[3]);
        const T v = T(m.vs), vf = v * F.v;
        g[0] = -(T(1) - vf * vf);
        g[1] = g[4] = -vf;
        g[5] = g[10] = g[15] = T(1);
        for (int q = 0; q < 3; ++q) {
            dg[16 * (q + 1)] = T(2) * v * v * F.v * F.d[q];
            dg[16 * (q + 1) + 1] = dg[16 * (q + 1) + 4] = -v * F.d[q];
        }
    }
}

}  // namespace sirius
