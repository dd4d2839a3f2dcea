// Pairs of floats (h + l, |l| <= ulp(h)/2) for the few values of an FP32 context that FP32 alone
// would lose: the internal energy rho e = rhoE - |rhoU|^2/(2 rho) and the pressure and temperature as
// offsets from the gauge state, and the gradient of the kinetic-energy objective. An FP64 warp
// instruction (a conversion too) holds its pipe for 16 clocks of an SM, an FP32 one for a quarter of a
// clock: the primitives' 21 in double kept the pipe busy for 50 to 60 % of k_prim and k_update, the
// gradient's 40 for half of k_adj_cell2. At 128^3: the objective stage's k_adj_cell2 about 200 -> 160 us,
// k_update 119 -> 115; k_prim 80 -> 52 us on the benchmark's state, and 72 with or without the pairs
// on a perturbed one, most of whose warps hold a value that the double form has to settle.
// The sums and products are the error-free transformations of Knuth and Dekker (T. J. Dekker, A
// floating-point technique for extending the available precision, Numer. Math. 18 (1971)): with
// u = 2^-24 a sum of pairs below errs by at most 3 u^2 of its operands' sizes, of a pair and a float by u^2 of
// the result's and the operand's, a product of pairs by 7 u^2 of its own and with a float by 2 u^2.
#pragma once
#include <math.h>
#include "physics.cuh"

namespace afvm {

// the roundings are spelled out: a contraction would break the error terms
#if defined(__CUDA_ARCH__)
AFVM_HD float f_add(float a, float b) { return __fadd_rn(a, b); }
AFVM_HD float f_mul(float a, float b) { return __fmul_rn(a, b); }
AFVM_HD float f_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
#else
AFVM_HD float f_add(float a, float b) { return a + b; }
AFVM_HD float f_mul(float a, float b) { return a * b; }
AFVM_HD float f_fma(float a, float b, float c) { return std::fma(a, b, c); }
#endif

// a + b, exactly; quick_sum: |a| >= |b|
AFVM_HD ff two_sum(float a, float b) {
    const float s = f_add(a, b), t = f_add(s, -a);
    return {s, f_add(f_add(a, -f_add(s, -t)), f_add(b, -t))};
}
AFVM_HD ff quick_sum(float a, float b) {
    const float s = f_add(a, b);
    return {s, f_add(b, -f_add(s, -a))};
}
// a b, exactly
AFVM_HD ff two_prod(float a, float b) {
    const float p = f_mul(a, b);
    return {p, f_fma(a, b, -p)};
}
AFVM_HD ff operator+(ff a, ff b) {
    const ff s = two_sum(a.h, b.h);
    return quick_sum(s.h, f_add(s.l, f_add(a.l, b.l)));
}
AFVM_HD ff operator+(ff a, float b) {
    const ff s = two_sum(a.h, b);
    return quick_sum(s.h, f_add(s.l, a.l));
}
AFVM_HD ff operator*(ff a, ff b) {
    const ff p = two_prod(a.h, b.h);
    return quick_sum(p.h, f_add(p.l, f_fma(a.h, b.l, f_mul(a.l, b.h))));
}
AFVM_HD ff operator*(ff a, float b) {
    const ff p = two_prod(a.h, b);
    return quick_sum(p.h, f_fma(a.l, b, p.l));
}
AFVM_HD ff operator-(ff a) { return {-a.h, -a.l}; }
// 1/a: a float reciprocal and one Newton step on the pair
AFVM_HD ff ff_rcp(ff a) {
    const float r = rcp(a.h);
    const float e = f_fma(-a.l, r, f_fma(-a.h, r, 1.0f));      // 1 - a r
    return quick_sum(r, f_mul(r, e));
}

// whether every value within e of the pair rounds to the same float (to a.h)
AFVM_HD bool rounds(ff a, float e) {
    return f_add(a.h, f_add(a.l, e)) == a.h && f_add(a.h, f_add(a.l, -e)) == a.h;
}

// what the pairs take: no term of theirs over- or underflows (NaN: no)
AFVM_HD bool ff_range(float x) { return x > 0x1p-40f && x < 0x1p40f; }

// pressure and temperature (gauge offsets) of a float state, rr = 1/rho in float as the velocities
// take it; false, with nothing written, where the pairs do not serve (the caller has the double form)
AFVM_HD bool prim_ff(const PhysFF& c, float rho, float r0, float r1, float r2, float rhoE, float rr, float* p, float* T) {
    const float most = fmaxf(fmaxf(fabsf(r0), fabsf(r1)), fabsf(r2));
    const ff q = two_prod(r0, r0) + two_prod(r1, r1) + two_prod(r2, r2);
    const ff ke = q * f_mul(0.5f, rr), e = -ke + rhoE;
    if (!(ff_range(rho) && ff_range(rhoE) && most < 0x1p40f && e.h > f_mul(0x1p-12f, rhoE))) return false;
    const ff pg = c.gm1 * e + -c.gP, Tg = e * rr * c.rCv + -c.gT;
    const float size = f_mul(0x1p-48f, f_fma(8.0f, ke.h, f_mul(14.0f, rhoE)));
    if (!(rounds(pg, f_mul(size, c.gm1.h)) && rounds(Tg, f_mul(f_mul(size, rr), c.rCv.h)))) return false;
    *p = pg.h;
    *T = Tg.h;
    return true;
}

// the gradient of obja rho |U|^2/2 V, rho = p/(Rg T), with respect to U, T and p (gauge offsets in
// v[0..4]), added to g[0..4]; false, with nothing written, as prim_ff (a dozen operations: 2^-40)
AFVM_HD bool kinetic_grad_ff(const PhysFF& c, ff obja, const float* v, float vol, float* g) {
    const ff T = two_sum(v[R_T], c.gT), p = two_sum(v[R_P], c.gP);
    const float most = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fabsf(v[2]));
    if (!(ff_range(fabsf(obja.h)) && ff_range(T.h) && ff_range(p.h) && ff_range(vol) && most < 0x1p40f)) return false;
    const ff rd = ff_rcp(T * c.Rg), rho = p * rd, w = obja * vol, wr = w * rho;
    const ff q = two_prod(v[0], v[0]) + two_prod(v[1], v[1]) + two_prod(v[2], v[2]);
    const ff h = w * (q * 0.5f) * rd;
    const ff add[5] = {wr * v[0], wr * v[1], wr * v[2], -(h * rho * c.Rg), h};
    for (int k = 0; k < 5; k++)
        if (!rounds(add[k], f_mul(0x1p-40f, fabsf(add[k].h)))) return false;
    for (int k = 0; k < 5; k++) g[k] = f_add(g[k], add[k].h);
    return true;
}

}  // namespace afvm
