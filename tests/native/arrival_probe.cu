// Leaves the arrival counts of the reductions where calls that overlapped may leave them. Test helper: compiled against libafvm.so by tests/test_gpu_arrival_count.py.
#include <cuda_runtime.h>
#include <string>
#include "ctx.cuh"

namespace afvm {
int sensitivity_launch(int nArrays, const double* const* grad, const double* const* pert, const int64_t* n,
                       double* partials, unsigned long long* arrived, unsigned long long call, double* out,
                       cudaStream_t s, std::string* err);
}

template <typename T>
static int set(T* p, T value) {
    if (!p) return 1;
    return cudaMemcpy(p, &value, sizeof(value), cudaMemcpyHostToDevice) == cudaSuccess ? 0 : 2;
}

// the reduction's third call on a scratch, whose second one has left its count `value` blocks further than
// it began; partials: 1024 x nArrays doubles, tail: the result and the count (device, two doubles).
// *out: the result
extern "C" int sensitivity_after(unsigned value, int nArrays, const double* const* grad, const double* const* pert,
                                 const int64_t* n, double* partials, double* tail, double* out) {
    unsigned long long* arrived = (unsigned long long*)(tail + 1);
    if (set(arrived, (2ull << 20) + value)) return 2;
    int st = afvm::sensitivity_launch(nArrays, grad, pert, n, partials, arrived, 3, tail, 0, nullptr);
    if (st) return st;
    return cudaMemcpy(out, tail, sizeof(double), cudaMemcpyDeviceToHost) == cudaSuccess ? 0 : 3;
}
// a context's own counts (present once the reduction, or the viscosity, has been called)
extern "C" int set_counters(afvm_ctx* ctx, unsigned value) {
    afvm::Ctx* c = reinterpret_cast<afvm::Ctx*>(ctx);
    int st = set((unsigned long long*)c->sensScratch, (c->sensCalls.load() << 20) + value);
    return st ? st : set((unsigned*)(c->viscWork + 48), value);
}
