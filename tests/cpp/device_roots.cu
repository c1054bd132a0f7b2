// The device's scalar reciprocals and roots (csrc/dual.cuh, csrc/roots.cuh) on arrays, and the warp drive's projection
// form at a radius, for tests/test_gpu_roots.py.
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
    inv_form(m, pos, F);
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
