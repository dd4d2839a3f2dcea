// Evaluates max_eig5, low and high (adfvm_gb300/csrc/eig5.cuh) on the device for host arrays. Test
// helper: compiled by tests/test_eig5_clusters.py.
#include <cuda_runtime.h>
#include "eig5.cuh"

__global__ void k_eig5(const double* a, int n, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s[5][5];
    for (int j = 0; j < 25; j++) s[j / 5][j % 5] = a[25 * (size_t)i + j];
    out[i] = afvm::max_eig5(s);
}
__global__ void k_low(const double* x, int n, float* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = afvm::low(x[i]);
}
__global__ void k_high(const float* x, int n, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = afvm::high(x[i]);
}

// out = kernel(in) over n items; 0 on success
template <typename X, typename Y>
static int run(void (*kernel)(const X*, int, Y*), const X* in, size_t per, int n, Y* out) {
    if (n <= 0 || n > (1 << 22)) return 1;
    X* x = nullptr;
    Y* y = nullptr;
    int st = 0;
    if (cudaMalloc(&x, sizeof(X) * per * n) != cudaSuccess || cudaMalloc(&y, sizeof(Y) * n) != cudaSuccess) st = 2;
    if (!st && cudaMemcpy(x, in, sizeof(X) * per * n, cudaMemcpyHostToDevice) != cudaSuccess) st = 3;
    if (!st) {
        kernel<<<(n + 127) / 128, 128>>>(x, n, y);
        if (cudaDeviceSynchronize() != cudaSuccess) st = 4;
    }
    if (!st && cudaMemcpy(out, y, sizeof(Y) * n, cudaMemcpyDeviceToHost) != cudaSuccess) st = 5;
    cudaFree(x);
    cudaFree(y);
    return st;
}
extern "C" int eig5_device(const double* a, int n, double* out) { return run(k_eig5, a, 25, n, out); }
extern "C" int low_device(const double* x, int n, float* out) { return run(k_low, x, 1, n, out); }
extern "C" int high_device(const float* x, int n, double* out) { return run(k_high, x, 1, n, out); }
