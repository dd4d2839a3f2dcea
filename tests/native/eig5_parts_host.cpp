// Host build of max_eig5 and its conversions low and high (adfvm_gb300/csrc/eig5.cuh). Test helper:
// compiled by tests/test_eig5_clusters.py.
#include <cmath>
#include "eig5.cuh"

extern "C" void eig5_host(const double* a, int n, double* out) {
    for (int i = 0; i < n; i++) out[i] = afvm::max_eig5(reinterpret_cast<const double(*)[5]>(a + 25 * (size_t)i));
}
extern "C" void low_host(const double* x, int n, float* out) {
    for (int i = 0; i < n; i++) out[i] = afvm::low(x[i]);
}
extern "C" void high_host(const float* x, int n, double* out) {
    for (int i = 0; i < n; i++) out[i] = afvm::high(x[i]);
}
