// The device's scalar reciprocals and roots (csrc/dual.cuh, csrc/roots.cuh) on arrays, for tests/test_gpu_roots.py.
#include <cuda_runtime.h>

#include "roots.cuh"

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
