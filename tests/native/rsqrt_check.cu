// Test helper: rsqrt64 of csrc/fp_bits.cuh on the device, for tests/test_rsqrt64.py.
#include <stdint.h>

#include "../../fastercap_gb300/csrc/fp_bits.cuh"

static __global__ void k_rsqrt64(int64_t n, const double *x, double *y) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = fcg::rsqrt64(x[i]);
}

// host arrays in and out; a CUDA error code
extern "C" int rsqrt64_all(int64_t n, const double *x, double *y) {
    double *d = nullptr;
    int e = (int)cudaMalloc((void **)&d, 2 * (size_t)n * sizeof(double));
    if (e) return e;
    e = (int)cudaMemcpy(d, x, (size_t)n * sizeof(double), cudaMemcpyHostToDevice);
    if (!e) {
        k_rsqrt64<<<256, 256>>>(n, d, d + n);
        e = (int)cudaGetLastError();
    }
    if (!e) e = (int)cudaMemcpy(y, d + n, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
