// The device's scalar reciprocals and roots (csrc/dual.cuh, csrc/roots.cuh) on arrays, the warp drive's projection form
// at a radius, and the two forms of the Kerr-Schild projection, for tests/test_gpu_roots.py and
// tests/test_gpu_naked_ring.py.
#include <cuda_runtime.h>

#include "roots.cuh"
#include "spacetime.cuh"

__global__ void apply(int f, long long n, const double* x, double* y) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    using namespace sirius;
    y[i] = f == 0   ? rcp_(v)
           : f == 1 ? rsqrt_(v)
           : f == 2 ? double(rcp_(float(v)))
           : f == 3 ? double(rsqrt_(float(v)))
           : f == 4 ? inv_root5(v)
                    : root_of_sum(v);
}

// radius and radial direction at x on the axis of motion of a warp drive, and the null value of a covector there before
// and after a projection
__global__ void warp_centre(sirius::MetricDev m, double x, double* y) {
    using namespace sirius;
    const double pos[4] = {0.0, x, 0.0, 0.0};
    double p[4] = {-1.0, 0.7, 0.3, -0.2};
    InvForm F;
    inv_form<true>(m, pos, F);
    y[0] = F.r;
    for (int i = 0; i < 4; ++i) y[1 + i] = i == 0 ? 0.0 : F.d[i];
    y[5] = project_null(m, F, p);
    for (int i = 0; i < 4; ++i) y[6 + i] = p[i];
}

extern "C" int device_warp_centre(double x, double* y) {
    sirius_metric s{};
    s.family = SIRIUS_METRIC_ALCUBIERRE;
    s.vs = 0.5; s.sigma = 8.0; s.R = 1.0;
    double* d = nullptr;
    cudaError_t e = cudaMalloc((void**)&d, 10 * sizeof(double));
    if (e != cudaSuccess) return int(e);
    warp_centre<<<1, 1>>>(sirius::metric_dev(s), x, d);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(y, d, 10 * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return int(e);
}

// state (x, p) -> 8 numbers: the momentum after the short projection, the null value before it, r; and the general one's
__global__ void ks_projections(sirius::MetricDev m, long long n, const double* state, double* fast, double* general) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    using namespace sirius;
    const double *x = state + 8 * i, *p = x + 4;
    double a[4], b[4], r;
    bool moved;
    for (int j = 0; j < 4; ++j) a[j] = b[j] = p[j];
    fast[8 * i + 4] = project_null_ks<double, true>(m, x, a, r, moved);
    InvForm F;
    inv_form<true>(m, x, F);
    general[8 * i + 4] = project_null(m, F, b);
    for (int j = 0; j < 4; ++j) {
        fast[8 * i + j] = a[j];
        general[8 * i + j] = b[j];
    }
    fast[8 * i + 5] = r;
    general[8 * i + 5] = F.r;
    for (int j = 6; j < 8; ++j) fast[8 * i + j] = general[8 * i + j] = 0.0;
}

extern "C" int device_ks_projections(const sirius_metric* s, long long n, const double* state, double* out) {
    double* d = nullptr;
    cudaError_t e = cudaMalloc((void**)&d, 3 * 8 * n * sizeof(double));
    if (e != cudaSuccess) return int(e);
    e = cudaMemcpy(d, state, 8 * n * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        ks_projections<<<unsigned((n + 127) / 128), 128>>>(sirius::metric_dev(*s), n, d, d + 8 * n, d + 16 * n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 8 * n, 16 * n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return int(e);
}

extern "C" int device_apply(int f, long long n, const double* x, double* y) {
    double* d = nullptr;
    cudaError_t e = cudaMalloc((void**)&d, 2 * n * sizeof(double));
    if (e != cudaSuccess) return int(e);
    e = cudaMemcpy(d, x, n * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        apply<<<unsigned((n + 255) / 256), 256>>>(f, n, d, d + n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(y, d + n, n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return int(e);
}
