// dual.cuh — register-resident forward-mode automatic differentiation.
//
// D3<T> carries a value and its gradient with respect to the three spatial
// coordinates of the integration chart. Metric potentials written with D3
// yield d_l g_{mu nu} without a tape or memory traffic: everything stays in
// registers and the compiler drops the zero tangents of constants. The
// reference's Dual<T> (src/Sirius.Core/Autodiff/MTDL001A.h:19-370) is a
// container whose tangent is never propagated; this type is the working form.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

// The metric templates compile for the device under nvcc and, in host-only
// translation units (the operation counter), as plain host code.
#ifndef SIRIUS_HD
#ifdef __CUDACC__
#define SIRIUS_HD __host__ __device__
#else
#define SIRIUS_HD
#endif
#endif

namespace sirius {

#ifdef __CUDACC__
// Reciprocal and roots used by the metric code.
//
// FP32: the special-function unit's approximations as they are (an approximation
// by design: the error budget of the FP32 path is set by the FP64 state and
// projection), without the subnormal scaling that the CUDA functions add around
// them; every normal argument gives the same bits either way.
//
// FP64: the unit's seeds (PTX rcp.approx.ftz.f64 and rsqrt.approx.ftz.f64) and one
// third-order Householder step, e the seed's residual:
//   1/x:        e = 1 - x y,    y <- y + y (e + e^2)
//   1/sqrt(x):  e = 1 - x y^2,  y <- y + y e (1/2 + 3/8 e)
// A seed good to 2^-20 leaves 2^-60, so a reciprocal is within 1.02 half-ulps and a reciprocal
// root, whose x y is rounded too, within 1.5, with no special-case branch beside each of the
// three per right-hand side (717 x 405 FP64 frame 5.78 -> 4.63 ms, 1024^2 mixed frame 20.3 ->
// 18.1 ms). The largest relative errors over 1e-300..1e300 are 1.1e-16 and 1.4e-16 (the CUDA
// functions': 1.1e-16 both). Arguments: normal numbers, for rcp_ of either sign, whose result is
// normal too; zero, a subnormal or an infinite argument gives NaN, so callers clamp theirs
// away from these where they can occur.
__device__ __forceinline__ float rcp_(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ double rcp_(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double rsqrt_(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-__dmul_rn(x, y), y, 1.0);
    return fma(__dmul_rn(y, e), fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ float sqrt_(float x) { return sqrtf(x); }
__device__ __forceinline__ double sqrt_(double x) { return sqrt(x); }
// Square root of a positive argument. FP32: x * rsqrt(x), two instructions with
// single-precision relative accuracy (the correctly rounded sqrtf is a longer
// sequence with a special-case branch); FP64: sqrt.
__device__ __forceinline__ float sqrtp_(float x) { return x * rsqrt_(x); }
__device__ __forceinline__ double sqrtp_(double x) { return sqrt(x); }
__device__ __forceinline__ float exp_(float x) { return __expf(x); }
__device__ __forceinline__ double exp_(double x) { return exp(x); }
__device__ __forceinline__ float tanh_(float x) { return tanhf(x); }
__device__ __forceinline__ double tanh_(double x) { return tanh(x); }
__device__ __forceinline__ void sincos_(float x, float& s, float& c) { sincosf(x, &s, &c); }
__device__ __forceinline__ void sincos_(double x, double& s, double& c) { sincos(x, &s, &c); }
#else
inline float rcp_(float x) { return 1.0f / x; }
inline double rcp_(double x) { return 1.0 / x; }
inline float sqrt_(float x) { return std::sqrt(x); }
inline double sqrt_(double x) { return std::sqrt(x); }
inline float rsqrt_(float x) { return 1.0f / std::sqrt(x); }
inline float sqrtp_(float x) { return std::sqrt(x); }
inline double sqrtp_(double x) { return std::sqrt(x); }
inline double rsqrt_(double x) { return 1.0 / std::sqrt(x); }
inline float exp_(float x) { return std::exp(x); }
inline double exp_(double x) { return std::exp(x); }
inline float tanh_(float x) { return std::tanh(x); }
inline double tanh_(double x) { return std::tanh(x); }
#endif

// Whether tanh(x) is exactly 1 in precision T: 1 - tanh(x) = 2 / (e^2x + 1) is below a
// quarter of the spacing under 1 (2^-26 in FP32, 2^-55 in FP64).
SIRIUS_HD __forceinline__ bool tanh_is_one(float x) { return x > 9.4f; }
SIRIUS_HD __forceinline__ bool tanh_is_one(double x) { return x > 19.5; }
template <class T>
SIRIUS_HD __forceinline__ bool tanh_is_one(T) { return false; }  // (an operation count takes the general path)

// a b + c in one rounding, and a product that no sum absorbs. Where a product meets a sum the
// compiler may fuse either or neither, by what surrounds it, and the kernels of one-frame
// launches and of batches (the same source, the metric in the parameter bank or in memory) then
// differ in last bits. The arithmetic of the FP64 and symplectic paths leaves it no choice.
template <class A, class B, class C>
SIRIUS_HD __forceinline__ auto fma_(A a, B b, C c) { return a * b + c; }
template <class A, class B>
SIRIUS_HD __forceinline__ auto mul_(A a, B b) { return a * b; }
#ifdef __CUDACC__
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
#endif

// The type of a function's constants when its variables are of type T.
template <class T>
struct scalar_of {
    using type = T;
};

// A value and its derivative along one direction: a function instantiated with D1
// gives its value and its Jacobian-vector product. Constants stay plain scalars
// (scalar_of), so nothing multiplies a zero tangent.
template <class T>
struct D1 {
    T v, d;
    D1() = default;
    SIRIUS_HD explicit D1(T value, T tangent = T(0)) : v(value), d(tangent) {}
};
template <class T>
struct scalar_of<D1<T>> {
    using type = T;
};
template <class T>
SIRIUS_HD __forceinline__ D1<T> operator+(D1<T> a, D1<T> b) { return D1<T>(a.v + b.v, a.d + b.d); }
template <class T>
SIRIUS_HD __forceinline__ D1<T> operator-(D1<T> a, D1<T> b) { return D1<T>(a.v - b.v, a.d - b.d); }
template <class T>
SIRIUS_HD __forceinline__ D1<T> operator*(D1<T> a, D1<T> b) { return D1<T>(a.v * b.v, a.d * b.v + a.v * b.d); }
template <class T>
SIRIUS_HD __forceinline__ D1<T> operator-(D1<T> a) { return D1<T>(-a.v, -a.d); }
template <class T>
SIRIUS_HD __forceinline__ D1<T> operator+(D1<T> a, T s) { return D1<T>(a.v + s, a.d); }
template <class T>
SIRIUS_HD __forceinline__ D1<T> operator+(T s, D1<T> a) { return a + s; }
template <class T>
SIRIUS_HD __forceinline__ D1<T> operator-(D1<T> a, T s) { return D1<T>(a.v - s, a.d); }
template <class T>
SIRIUS_HD __forceinline__ D1<T> operator-(T s, D1<T> a) { return D1<T>(s - a.v, -a.d); }
template <class T>
SIRIUS_HD __forceinline__ D1<T> operator*(T s, D1<T> a) { return D1<T>(s * a.v, s * a.d); }
template <class T>
SIRIUS_HD __forceinline__ D1<T> operator*(D1<T> a, T s) { return s * a; }
template <class T>
SIRIUS_HD __forceinline__ D1<T>& operator+=(D1<T>& a, D1<T> b) { a = a + b; return a; }
template <class T>
SIRIUS_HD __forceinline__ D1<T>& operator-=(D1<T>& a, D1<T> b) { a = a - b; return a; }
template <class T>
SIRIUS_HD __forceinline__ D1<T> rcp_(D1<T> a) {
    const T y = rcp_(a.v);
    return D1<T>(y, -y * y * a.d);
}
template <class T>
SIRIUS_HD __forceinline__ D1<T> rsqrt_(D1<T> a) {
    const T y = rsqrt_(a.v);
    return D1<T>(y, T(-0.5) * y * y * y * a.d);
}

template <class T>
struct D3 {
    T v;
    T d[3];
};

template <class T>
SIRIUS_HD __forceinline__ D3<T> dconst(T v) {
    return D3<T>{v, {T(0), T(0), T(0)}};
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> dvar(T v, int axis) {
    D3<T> r{v, {T(0), T(0), T(0)}};
    r.d[axis] = T(1);
    return r;
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> operator+(const D3<T>& a, const D3<T>& b) {
    return D3<T>{a.v + b.v, {a.d[0] + b.d[0], a.d[1] + b.d[1], a.d[2] + b.d[2]}};
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> operator-(const D3<T>& a, const D3<T>& b) {
    return D3<T>{a.v - b.v, {a.d[0] - b.d[0], a.d[1] - b.d[1], a.d[2] - b.d[2]}};
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> operator-(const D3<T>& a) {
    return D3<T>{-a.v, {-a.d[0], -a.d[1], -a.d[2]}};
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> operator+(const D3<T>& a, T s) {
    return D3<T>{a.v + s, {a.d[0], a.d[1], a.d[2]}};
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> operator-(const D3<T>& a, T s) {
    return D3<T>{a.v - s, {a.d[0], a.d[1], a.d[2]}};
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> operator*(const D3<T>& a, T s) {
    return D3<T>{a.v * s, {a.d[0] * s, a.d[1] * s, a.d[2] * s}};
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> operator*(T s, const D3<T>& a) {
    return a * s;
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> operator*(const D3<T>& a, const D3<T>& b) {
    return D3<T>{a.v * b.v,
                 {a.d[0] * b.v + a.v * b.d[0], a.d[1] * b.v + a.v * b.d[1], a.d[2] * b.v + a.v * b.d[2]}};
}
// 1/a
template <class T>
SIRIUS_HD __forceinline__ D3<T> inv(const D3<T>& a) {
    const T r = rcp_(a.v);
    const T r2 = -r * r;
    return D3<T>{r, {a.d[0] * r2, a.d[1] * r2, a.d[2] * r2}};
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> operator/(const D3<T>& a, const D3<T>& b) {
    return a * inv(b);
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> dsqrt(const D3<T>& a) {
    const T s = sqrt_(a.v);
    const T h = T(0.5) * rcp_(s);
    return D3<T>{s, {a.d[0] * h, a.d[1] * h, a.d[2] * h}};
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> dexp(const D3<T>& a) {
    const T e = exp_(a.v);
    return D3<T>{e, {a.d[0] * e, a.d[1] * e, a.d[2] * e}};
}
template <class T>
SIRIUS_HD __forceinline__ D3<T> dtanh(const D3<T>& a) {
    const T t = tanh_(a.v);
    const T s = T(1) - t * t;
    return D3<T>{t, {a.d[0] * s, a.d[1] * s, a.d[2] * s}};
}
// a with its gradient replaced by g (the chain-rule seed of an implicit function)
template <class T>
SIRIUS_HD __forceinline__ D3<T> dwith(T v, T g0, T g1, T g2) {
    return D3<T>{v, {g0, g1, g2}};
}

}  // namespace sirius
