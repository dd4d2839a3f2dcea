// Host build of the pairs of floats (adfvm_gb300/csrc/ff32.cuh). Test helper: compiled by
// tests/test_ff32.py.
#include <cmath>
#include "ff32.cuh"

using namespace afvm;

static Phys phys(const double* c) {
    Phys P = {};
    P.gm1 = c[0]; P.Cv = c[1]; P.rCv = 1.0 / c[1];
    P.gaugeP = c[2]; P.gaugeT = c[3];
    P.gamma = 1.0 + c[0]; P.Cp = P.gamma * P.Cv;
    finish_phys(P);
    return P;
}
// state rho, rhoU (3), rhoE and 1/rho -> p, T; ok: whether the pairs took it
extern "C" void ff_prims(const double* c, const float* s, int n, float* pT, int* ok) {
    const Phys P = phys(c);
    for (int i = 0; i < n; i++, s += 6, pT += 2)
        ok[i] = prim_ff(P.pair, s[0], s[1], s[2], s[3], s[4], s[5], pT, pT + 1);
}
// prims U (3), T, p and the volume -> the five terms added to g
extern "C" void ff_kinetic(const double* c, double obja, const float* s, int n, float* g, int* ok) {
    const Phys P = phys(c);
    for (int i = 0; i < n; i++, s += 6, g += 5) ok[i] = kinetic_grad_ff(P.pair, ff_of(obja), s, s[5], g);
}
