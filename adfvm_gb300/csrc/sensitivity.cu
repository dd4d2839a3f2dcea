// Sensitivity dot product sum_k <grad_k, pert_k> in FP64 (cmesh.computeSensitivity,
// adFVM/cpp/cmesh.cpp:309-340, an OpenMP reduction in the reference).
//
// Deterministic two-level reduction in one launch for up to SENS_PACK arrays: an array's blocks
// (at most SENS_BLOCKS) run a grid-stride loop over it and write one partial sum each; the last
// block of the launch to arrive adds all of them in a fixed order. The result does not depend on
// timing, and repeated calls give identical bits. The arrays' addresses and sizes travel as kernel
// arguments and the context's result lands in mapped host memory, so a call is one launch and one
// wait. With a launch an array, one for the sum and a copy each way a call took 38 us of the stream
// and more of the host: the 128x64 cylinder's ten-step FP64 sweep, ten calls with three arrays,
// 4.67 -> 4.26 ms.
#include <cuda_runtime.h>
#include <atomic>
#include <mutex>
#include "ctx.cuh"

namespace afvm {

constexpr int SENS_BLOCKS = 1024;
constexpr int SENS_PACK = 16;

__device__ __forceinline__ double warp_sum(double v) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    return v;
}

struct SensPack {
    const double *g[SENS_PACK], *p[SENS_PACK];
    long long n[SENS_PACK];
    int first[SENS_PACK + 1];      // the first block of each array
    int arrays;
};

__device__ __forceinline__ double sens_block_sum(double v, double* sh) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x < 32) r = warp_sum((threadIdx.x < BLOCK / 32) ? sh[threadIdx.x] : 0.0);
    __syncthreads();
    return r;
}

// The arrival count is never cleared: a call counts from SENS_CALL times its number, to which each of its
// blocks first raises the count (it is lower, from the call before). Calls that overlap spoil one
// another's results, and leave the count at a value that serves the next call as well.
constexpr unsigned long long SENS_CALL = 1ull << 20;
static_assert(SENS_PACK * SENS_BLOCKS < SENS_CALL, "a launch's blocks");

// this launch's partials follow the base ones of the launches before; total: all of them, summed
// into *out by the last launch's last block (out NULL: not the last launch). from: the call's count
__global__ void __launch_bounds__(BLOCK) k_sens(SensPack a, double* partials, int base, int total,
                                                unsigned long long* arrived, unsigned long long from, double* out) {
    __shared__ double sh[BLOCK / 32];
    __shared__ bool last;
    if (out && threadIdx.x == 0) atomicMax(arrived, from);
    int k = 0;
    while (k + 1 < a.arrays && (int)blockIdx.x >= a.first[k + 1]) k++;
    const double* __restrict__ g = a.g[k];
    const double* __restrict__ p = a.p[k];
    const long long n = a.n[k], step = (long long)(a.first[k + 1] - a.first[k]) * BLOCK;
    double v = 0.0;
    for (long long i = ((int)blockIdx.x - a.first[k]) * (long long)BLOCK + threadIdx.x; i < n; i += step) v += g[i] * p[i];
    double r = sens_block_sum(v, sh);
    if (threadIdx.x == 0) {
        partials[base + blockIdx.x] = r;
        __threadfence();
        last = out && atomicAdd(arrived, 1ull) == from + gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    v = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < total; i += BLOCK) v += __ldcg(partials + i);
    r = sens_block_sum(v, sh);
    if (threadIdx.x == 0) *out = r;
}

static int sens_blocks(long long n) {
    long long b = (n + BLOCK - 1) / BLOCK;
    return (int)(b < SENS_BLOCKS ? b : SENS_BLOCKS);
}

// queues the reduction of nArrays arrays; partials: SENS_BLOCKS x nArrays; arrived: the scratch's arrival
// count, zero before its first call; call: the number of this call on the scratch, from 1
int sensitivity_launch(int nArrays, const double* const* grad, const double* const* pert, const int64_t* n,
                       double* partials, unsigned long long* arrived, unsigned long long call, double* out,
                       cudaStream_t s, std::string* err) {
    for (int k = 0; k < nArrays; k++)
        if (n[k] < 0 || (n[k] > 0 && (!grad[k] || !pert[k]))) {
            if (err) *err = "afvm_sensitivity: array " + std::to_string(k) + " has a bad size or pointer";
            return AFVM_ERR_BAD_ARG;
        }
    int base = 0;
    for (int k0 = 0; k0 < nArrays; k0 += SENS_PACK) {
        const int m = nArrays - k0 < SENS_PACK ? nArrays - k0 : SENS_PACK;
        SensPack a = {};
        a.arrays = m;
        for (int k = 0; k < m; k++) {
            a.g[k] = grad[k0 + k];
            a.p[k] = pert[k0 + k];
            a.n[k] = n[k0 + k];
            a.first[k + 1] = a.first[k] + sens_blocks(n[k0 + k]);
        }
        const bool end = k0 + m == nArrays;
        // (one block at the end even when its arrays are empty: it writes the sum)
        const int blocks = a.first[m] > 0 ? a.first[m] : (end ? 1 : 0);
        if (!blocks) continue;
        if (a.first[m] == 0) a.first[m] = 1;
        k_sens<<<blocks, BLOCK, 0, s>>>(a, partials, base, base + blocks, arrived, call * SENS_CALL,
                                         end ? out : nullptr);
        base += blocks;
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        if (err) *err = std::string("afvm_sensitivity: ") + cudaGetErrorString(e);
        return AFVM_ERR_CUDA;
    }
    return AFVM_OK;
}

int sensitivity_dev(Ctx* c, int nArrays, const double* const* grad, const double* const* pert, const int64_t* n,
                    double* out, cudaStream_t s) {
    if (nArrays <= 0 || !grad || !pert || !n || !out) return fail(c, AFVM_ERR_BAD_ARG, "afvm_sensitivity arguments");
    // scratch sized for this call, kept on the context and grown on demand
    size_t need = sizeof(double) * ((size_t)nArrays * SENS_BLOCKS + 1);
    if (need > c->sensBytes) {
        if (c->sensScratch) cudaFree(c->sensScratch);
        c->sensScratch = nullptr;
        c->sensBytes = 0;
        if (cudaMalloc(&c->sensScratch, need) != cudaSuccess) {
            cudaGetLastError();
            return fail(c, AFVM_ERR_OOM, "afvm_sensitivity scratch");
        }
        c->sensBytes = need;
        cudaError_t e = cudaMemsetAsync(c->sensScratch, 0, sizeof(double), s);
        if (e != cudaSuccess) return cuda_fail(c, e, "afvm_sensitivity scratch");
    }
    ProfScope ps(c, KID_SENS, s);
    int st = sensitivity_launch(nArrays, grad, pert, n, (double*)c->sensScratch + 1, (unsigned long long*)c->sensScratch,
                                ++c->sensCalls, c->hostOutDev + 2, s, &c->err);
    if (st) return st;
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(c, e, "afvm_sensitivity result");
    *out = c->hostOut[2];
    return AFVM_OK;
}

// ---------------------------------------------------------------------------------------
// Allocation-free variant (afvm_sensitivity_noalloc).
//
// Some callers may not allocate device memory: an application that gives this library a
// fixed share of the GPU up front and makes every allocation itself, or a plug-in loaded
// into a host program whose memory pool it must not touch. Such a caller can create no
// context and cannot let afvm_sensitivity grow its scratch. For them the reduction's
// scratch (block partials, the result and the arrival count) is this file-scope device array,
// sized for at most AFVM_SENSITIVITY_NOALLOC_MAX_ARRAYS arrays. Every GPU that loads the library
// keeps it (~129 KB) until the process exits. All calls share it: two calls that overlap on the
// GPU (different streams, or different host threads without ordering) race on it.
// ---------------------------------------------------------------------------------------

constexpr int NOALLOC_MAX_ARRAYS = AFVM_SENSITIVITY_NOALLOC_MAX_ARRAYS;
constexpr size_t NOALLOC_PARTIALS = (size_t)NOALLOC_MAX_ARRAYS * SENS_BLOCKS;
// partials, then the result, then the arrival count (zero when the library is loaded)
constexpr size_t NOALLOC_DOUBLES = NOALLOC_PARTIALS + 2;

static __device__ __align__(256) double g_sens_noalloc_scratch[NOALLOC_DOUBLES];

// Host code must not use the symbol itself as a device address: the device address of the
// array is looked up by the first call on each device, with that device current, and cached
// here (so that first call belongs before any stream capture). cudaDeviceReset unloads the
// module: the cached address is then stale, and calls after a reset are not supported.
static std::mutex g_noalloc_mutex;
static double* g_noalloc_ptr[256] = {nullptr};
static std::atomic<unsigned long long> g_noalloc_calls{0};     // (on any device)

static int noalloc_scratch(int device, double** out) {
    if (device < 0 || device >= 256) return AFVM_ERR_BAD_ARG;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[device]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_sens_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            cudaGetLastError();
            return AFVM_ERR_CUDA;
        }
        g_noalloc_ptr[device] = (double*)p;
    }
    *out = g_noalloc_ptr[device];
    return AFVM_OK;
}

}  // namespace afvm

extern "C" int afvm_sensitivity_noalloc(int32_t device, int32_t nArrays, const double* const* grad,
                                        const double* const* pert, const int64_t* n, double* out, void* stream) {
    using namespace afvm;
    if (nArrays <= 0 || nArrays > NOALLOC_MAX_ARRAYS || !grad || !pert || !n || !out) return AFVM_ERR_BAD_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return AFVM_ERR_BAD_ARG;
    }
    // every array must be memory of `device` and the stream a stream of it: a host pointer or
    // another GPU's memory would make the kernels fault or read the wrong memory
    for (int k = 0; k < nArrays; k++) {
        if (n[k] <= 0) continue;
        const void* ptrs[2] = {grad[k], pert[k]};
        for (const void* q : ptrs) {
            cudaPointerAttributes a;
            if (!q || cudaPointerGetAttributes(&a, q) != cudaSuccess ||
                (a.type != cudaMemoryTypeDevice && a.type != cudaMemoryTypeManaged) || a.device != device) {
                cudaGetLastError();
                return AFVM_ERR_BAD_ARG;
            }
        }
    }
    if (stream) {
        int sdev = -1;
        if (cudaStreamGetDevice((cudaStream_t)stream, &sdev) != cudaSuccess || sdev != device) {
            cudaGetLastError();
            return AFVM_ERR_BAD_ARG;
        }
    }
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != device && cudaSetDevice(device) != cudaSuccess) {
        cudaGetLastError();
        return AFVM_ERR_CUDA;
    }
    double* scratch = nullptr;
    int st = noalloc_scratch(device, &scratch);
    if (st == AFVM_OK) {
        double* partials = scratch;
        double* result = scratch + NOALLOC_PARTIALS;
        cudaStream_t s = (cudaStream_t)stream;
        // every partial read below is written earlier in this call, so nothing left by a previous
        // call is used and nothing needs clearing
        st = sensitivity_launch(nArrays, grad, pert, n, partials, (unsigned long long*)(result + 1), ++g_noalloc_calls,
                                result, s, nullptr);
        if (st == AFVM_OK && (cudaStreamSynchronize(s) != cudaSuccess ||
                              cudaMemcpy(out, result, sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)) {
            cudaGetLastError();
            st = AFVM_ERR_CUDA;
        }
    }
    if (prev >= 0 && prev != device) cudaSetDevice(prev);
    return st;
}
