// Evaluates the library's integer-pipe FP64 product, reciprocal and reciprocal square root
// (soft_mul, soft_rcp, soft_rsqrt in adfvm_gb300/csrc/soft64.cuh) and the out-of-window flag of
// the latter two for host arrays. Test helper: compiled by tests/test_gpu_soft64.py.
#include <cuda_runtime.h>
#include "soft64.cuh"

__global__ void k_probe(const double* x, const double* y, double* out, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    using namespace afvm;
    out[i] = soft_mul(x[i], y[i]);
    soft_flag() = 0;
    out[n + i] = soft_rcp<64>(x[i]);
    out[2 * n + i] = soft_flag();
    soft_flag() = 0;
    out[3 * n + i] = soft_rsqrt(x[i]);
    out[4 * n + i] = soft_flag();
}

extern "C" int soft64_probe(const double* x, const double* y, double* out, int n) {
    if (n <= 0 || n > (1 << 26)) return 1;
    double* d = nullptr;
    size_t b = sizeof(double) * (size_t)n;
    if (cudaMalloc(&d, 7 * b) != cudaSuccess) return 2;
    int st = 0;
    if (cudaMemcpy(d, x, b, cudaMemcpyHostToDevice) != cudaSuccess) st = 3;
    if (!st && cudaMemcpy(d + n, y, b, cudaMemcpyHostToDevice) != cudaSuccess) st = 3;
    if (!st) {
        k_probe<<<(n + 127) / 128, 128>>>(d, d + n, d + 2 * (size_t)n, n);
        if (cudaDeviceSynchronize() != cudaSuccess) st = 4;
    }
    if (!st && cudaMemcpy(out, d + 2 * (size_t)n, 5 * b, cudaMemcpyDeviceToHost) != cudaSuccess) st = 5;
    cudaFree(d);
    return st;
}
