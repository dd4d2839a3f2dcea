// Adjoint stabilisation by artificial viscosity (adFVM/postpro.py:491-718 with the compiled
// helpers of adFVM/cpp/scaling.cpp:84-159 and the heat equation of matop_petsc.cpp:230-372).
//
// For a primal state u:
//   k_visc_sound  per cell and ghost: the sound speed (once, not for every face that reads it)
//   k_visc_cell   per cell, gathered over its faces in the reference's collate order: face
//                 values (central on internal and coupled faces, the ghost value on other
//                 boundary faces) -> gradU, divU = tr gradU, gradp, gradc (op.grad / op.div); the
//                 5x5 symmetriser M of the 'turkel' or 'abarbanel' kind, MS = (M + M^T)/2, and its
//                 largest eigenvalue (eig5.cuh); 'uniform' is 1. The norm sum M^2 V in its last block.
//   k_visc_face   M <- scaling M / sqrt(sum M^2 V / sum V), ghost values of the default boundary
//                 (the ghost's source cell); per face DT = w M_own + (1-w) M_nbr and the
//                 coefficient dt A DT / delta of the implicit heat equation.
// and the adjoint fields a (plain gradients) are replaced by V x, where x solves, for each of
// the 5 components,
//   V_c x_c + sum_k dt A_k DT_k / delta_k (x_c - x_nbr(k)) = V_c (a_c / V_c)
// over the faces k of c with an internal neighbour - the symmetric form of the reference's
// (1 + sum coef) x_c - sum coef x_nbr = x0_c, coef = dt A DT / (delta V_c). It is solved by
// preconditioned conjugate gradients (Jacobi preconditioner), the five components in lockstep,
// to a relative residual of 1e-13 (the reference: 1000 Jacobi sweeps on the GPU or GMRES
// through PETSc on the CPU). Everything here is FP64 whatever the context's precision.
//
// The FP64 pipe binds every kernel here, so their FP64 instructions are what was cut: divisions are
// products with reciprocals formed once (with the remainder taken back where a result depends on
// them: quotient), alpha and beta are formed once an iteration by the last block of the kernel that
// sums their dot products (which also spares the single-block kernels in between), and a block adds
// its 5 or 10 dot products through shared memory (about 8 FP64 instructions a warp and product
// instead of 12 in every warp). An iteration is three kernels.
// Vectors are interleaved, five components a cell: a neighbour's are in two sectors instead of five.
// 262,144 cells in FP64, four iterations: 3.27 -> 0.89 ms (k_visc_cell 2.13 -> 0.31, an iteration
// 198 -> 87 us: q = A p 57 + 10 -> 44, update 84 + 17.5 + 2 -> 32, direction 27.5 -> 11).
#include <cuda_runtime.h>
#include <math.h>
#include <algorithm>
#include "ctx.cuh"
#include "eig5.cuh"

namespace afvm {

namespace {

constexpr double UREF = 33., PREF = 1e5;   // RCF reference scales (adFVM/density.py:57-59)

constexpr int VT = 128;                    // threads a block of the kernels here

// Adds the K values of every thread of the block and, in the last block of the grid to arrive,
// the blocks' sums: true there in thread 0, with the grid's sums in out (the order of every
// addition is fixed). partials: K x gridDim.x; arrived: zero before the first launch and after
// each (cleared at the start of a call).
template <int K>
__device__ __forceinline__ bool grid_sums(const double* v, double* partials, unsigned* arrived, double* out) {
    __shared__ double sh[K * VT];
    __shared__ bool last;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nb = gridDim.x;
    for (int k = 0; k < K; k++) sh[k * VT + t] = v[k];
    __syncthreads();
    for (int k = warp; k < K; k += VT / 32) {
        double s = (sh[k * VT + lane] + sh[k * VT + 32 + lane]) + (sh[k * VT + 64 + lane] + sh[k * VT + 96 + lane]);
        for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
        if (lane == 0) partials[(size_t)k * nb + blockIdx.x] = s;
    }
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicInc(arrived, nb - 1) == (unsigned)(nb - 1);
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double s[K];
    for (int k = 0; k < K; k++) s[k] = 0.0;
    for (int i = t; i < nb; i += VT)
        for (int k = 0; k < K; k++) s[k] += __ldcg(partials + (size_t)k * nb + i);
    for (int k = 0; k < K; k++) sh[k * VT + t] = s[k];
    __syncthreads();
    for (int k = warp; k < K; k += VT / 32) {
        double w = (sh[k * VT + lane] + sh[k * VT + 32 + lane]) + (sh[k * VT + 64 + lane] + sh[k * VT + 96 + lane]);
        for (int off = 16; off > 0; off >>= 1) w += __shfl_down_sync(0xffffffffu, w, off);
        if (lane == 0) sh[k * VT] = w;
    }
    __syncthreads();
    if (t != 0) return false;
    for (int k = 0; k < K; k++) out[k] = sh[k * VT];
    return true;
}

// x / y and sqrt(x) rounded once, from products with r = 1/y and r = 1/sqrt(x): the product rounds a
// second time, the remainder takes that back (two FP64 instructions)
__device__ __forceinline__ double quotient(double x, double y, double r) {
    const double q = x * r;
    return fma(fma(-q, y, x), r, q);
}
__device__ __forceinline__ double root(double x, double r) {
    const double s = x * r;
    return fma(fma(-s, s, x), 0.5 * r, s);
}

template <typename R>
__global__ void __launch_bounds__(VT) k_visc_sound(MeshDev<R> m, Phys P, const R* __restrict__ rec,
                                                   double* __restrict__ snd) {
    const int c = blockIdx.x * VT + threadIdx.x;
    if (c >= m.nC) return;
    const double c2 = (P.gamma * rec_T<R>(P, rec[(size_t)c * REC + R_T])) * (P.Cp - P.Cv);
    snd[c] = c2 == 0.0 ? 0.0 : root(c2, rsqrt_(c2));
}

template <typename R>
__global__ void __launch_bounds__(VT) k_visc_cell(MeshDev<R> m, Phys P, const R* __restrict__ rec,
                                                  const double* __restrict__ snd, int kind, double Vt, double scaling,
                                                  double* __restrict__ M, double* partials, unsigned* arrived,
                                                  double* fac) {
    const int c = blockIdx.x * VT + threadIdx.x;
    double contrib = 0.0;
    if (c < m.nIC) {
        const size_t n = m.nIC;
        const size_t nF = m.nF;
        double val = 1.0;
        if (kind != AFVM_VISC_UNIFORM) {
            const double g = P.gamma;
            double gU[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, gp[3] = {0, 0, 0}, gc[3] = {0, 0, 0};
            for (int k = 0; k < 6; k++) {
                const int e = m.accf[k * n + c];
                const double wt = m.accw[k * n + c];
                const bool ownerSide = e >= 0;
                const int f = ownerSide ? e : ~e;
                const int iN = m.nbr[f];
                const R* rN = rec + (size_t)iN * REC;
                double UF[3], pF, cF;
                if (f < m.nIF || m.fkind[f - m.nIF] == FACE_COUPLED) {
                    const int iO = m.own[f];
                    const R* rO = rec + (size_t)iO * REC;
                    const double w = m.wts[f], w1 = 1 - w;
                    for (int i = 0; i < 3; i++) UF[i] = (double)rO[i] * w + (double)rN[i] * w1;
                    pF = (double)rO[R_P] * w + (double)rN[R_P] * w1;
                    cF = snd[iN] * w1 + snd[iO] * w;
                } else {
                    for (int i = 0; i < 3; i++) UF[i] = rN[i];
                    pF = rN[R_P];
                    cF = snd[iN];
                }
                const double sw = ownerSide ? wt : -wt;
                for (int j = 0; j < 3; j++) {
                    const double N = (double)m.nrm[j * nF + f] * sw;
                    for (int i = 0; i < 3; i++) gU[i][j] += UF[i] * N;
                    gp[j] += pF * N;
                    gc[j] += cF * N;
                }
            }
            // FP32 records hold p - gaugeP: the sum above missed gaugeP times the cell's sum of A/V N
            // (zero when the cell's face area vectors close, not for warped faces)
            if constexpr (kGauge<R>)
                for (int j = 0; j < 3; j++) gp[j] += P.gaugeP * m.gclD[j * n + c];
            const double dU = gU[0][0] + gU[1][1] + gU[2][2];
            const R* r = rec + (size_t)c * REC;
            const double T = rec_T<R>(P, r[R_T]), p = rec_p<R>(P, r[R_P]);
            // (each entry rounds no more often than with divisions: quotient, root)
            const double g1 = g - 1, e = (P.Cv * T) * g1;
            const double rho = quotient(p, e, rcp(e)), rrho = rcp(rho), rp = rcp(p);
            const double c2 = quotient(g * p, rho, rrho), rc = rsqrt_(c2), cc = root(c2, rc);
            const double rhoc = rho * cc, rrc = rrho * rc;
            // grad rho = g (grad p - c p) / c^2
            double gs[3];
            for (int j = 0; j < 3; j++) gs[j] = gp[j] - cc * p;
            double A[5][5];
            for (int i = 0; i < 5; i++)
                for (int j = 0; j < 5; j++) A[i][j] = 0.0;
            // M = M1/2 - M2 (postpro.py:571-602)
            if (kind == AFVM_VISC_TURKEL) {
                const double gpr = (g * p) * rho;
                const double pg = quotient(PREF / (2 * UREF), gpr, rcp(g) * (rp * rrho));
                for (int i = 0; i < 5; i++) A[i][i] = dU / 2;
                for (int j = 0; j < 3; j++) { A[0][1 + j] += gc[j] / 2; A[1 + j][0] += gc[j] / 2; }
                A[0][0] -= g1 * dU / 2;
                for (int j = 0; j < 3; j++) {
                    const double q = quotient(gp[j], rhoc, rrc);
                    A[0][1 + j] -= q;
                    A[1 + j][0] -= (0.5 * g1) * q;
                    A[1 + j][4] -= gp[j] * pg;
                    A[4][1 + j] -= (gp[j] - g * gs[j]) * (UREF / PREF);
                    for (int k = 0; k < 3; k++) A[1 + j][1 + k] -= gU[j][k];
                }
                A[0][4] -= quotient(dU * (PREF / (2 * UREF)), rhoc, rrc);
                A[4][4] -= g1 * dU / 2;
            } else {
                const double rsg = rsqrt_(g), sg = root(g, rsg), sg1 = root(g1, rsqrt_(g1)), rg1 = rcp(g1);
                const double a = sg1 * quotient(cc, sg, rsg);
                double gb[3], ga[3];
                for (int j = 0; j < 3; j++) { gb[j] = quotient(gc[j], sg, rsg); ga[j] = gb[j] * sg1; }
                for (int i = 0; i < 5; i++) A[i][i] = dU / 2;
                for (int j = 0; j < 3; j++) {
                    A[0][1 + j] += gb[j] / 2; A[1 + j][0] += gb[j] / 2;
                    A[1 + j][4] += ga[j] / 2; A[4][1 + j] += ga[j] / 2;
                }
                for (int j = 0; j < 3; j++) {
                    A[0][1 + j] -= quotient(gs[j] * sg, rhoc, rrc);      // b grad rho / rho, b = c / sqrt(g)
                    A[1 + j][4] -= 0.5 * quotient(a * gp[j], p, rp);
                    A[4][1 + j] -= 2 * quotient(ga[j], g1, rg1);
                    for (int k = 0; k < 3; k++) A[1 + j][1 + k] -= gU[j][k];
                }
                A[0][4] -= sg1 * dU / 2;
                A[4][4] -= g1 * dU / 2;
            }
            // MS = (M + M^T)/2, upper triangle
            double S[5][5];
            for (int i = 0; i < 5; i++)
                for (int j = i; j < 5; j++) S[i][j] = (A[i][j] + A[j][i]) / 2;
            val = max_eig5(S);
        }
        M[c] = val;
        contrib = val * val * (double)m.vol[c];
    }
    double s;
    if (grid_sums<1>(&contrib, partials, arrived, &s)) fac[0] = scaling / sqrt(s / Vt);
}

// the scaled viscosity of every cell and ghost, for a caller that asks for it
template <typename R>
__global__ void __launch_bounds__(VT) k_visc_scaled(MeshDev<R> m, const double* __restrict__ M,
                                                    const double* __restrict__ fac, double* __restrict__ out) {
    const int c = blockIdx.x * VT + threadIdx.x;
    if (c < m.nC) out[c] = M[c < m.nIC ? c : m.gsrc[c - m.nIC]] * fac[0];
}

// per face DT = w M_own + (1-w) M_nbr of the scaled viscosity and the heat-equation coefficient
// dt A DT / delta
template <typename R>
__global__ void __launch_bounds__(VT) k_visc_face(MeshDev<R> m, const double* __restrict__ M,
                                                  const double* __restrict__ fac, double dt, double* __restrict__ DT,
                                                  double* __restrict__ coef) {
    const int f = blockIdx.x * VT + threadIdx.x;
    if (f >= m.nF) return;
    const double w = m.wts[f], s = fac[0];
    const int iN = f < m.nIF ? m.nbr[f] : m.gsrc[f - m.nIF];
    const double d = (M[m.own[f]] * s) * w + (M[iN] * s) * (1 - w);
    DT[f] = d;
    const double dlt = m.dlt[f];
    coef[f] = dt * quotient((double)m.area[f] * d, dlt, rcp(dlt));
}

// ---- PCG on (V + dt L) x = a, five right-hand sides in lockstep; vectors are n x 5
//
// sc: [0..5) r.z, [5..10) alpha, [10..15) beta, [15..20) r.r, [20..25) |rhs|^2

// the right-hand side V (a / V) = a (the symmetric form's: the adjoint field itself), x0 = a / V
template <typename R, typename S>
__global__ void __launch_bounds__(VT) k_heat_rhs(MeshDev<R> m, const S* __restrict__ ar, const S* __restrict__ au,
                                                 const S* __restrict__ ae, double* __restrict__ x, double* partials,
                                                 unsigned* arrived, double* sc) {
    double v[5] = {0, 0, 0, 0, 0};
    for (int c = blockIdx.x * VT + threadIdx.x; c < m.nIC; c += gridDim.x * VT) {
        const double a[5] = {(double)ar[c], (double)au[3 * c], (double)au[3 * c + 1], (double)au[3 * c + 2], (double)ae[c]};
        const double V = m.vol[c], rV = rcp(V);
        for (int q = 0; q < 5; q++) {
            x[5 * (size_t)c + q] = quotient(a[q], V, rV);
            v[q] += a[q] * a[q];
        }
    }
    double s[5];
    if (grid_sums<5>(v, partials, arrived, s))
        for (int q = 0; q < 5; q++) sc[20 + q] = s[q];
}

// the matrix by cell (the volume, the diagonal's reciprocal, and per slot the neighbour and its weight:
// the cell itself and zero across a boundary), r = a - A x0, p = z = r / diagonal, r.z and r.r
template <typename R, typename S>
__global__ void __launch_bounds__(VT) k_heat_init(MeshDev<R> m, const double* __restrict__ coef,
                                                  const S* __restrict__ ar, const S* __restrict__ au,
                                                  const S* __restrict__ ae, const double* __restrict__ x,
                                                  double* __restrict__ vol, double* __restrict__ rdiag,
                                                  double* __restrict__ wgt, int* __restrict__ nbh,
                                                  double* __restrict__ r, double* __restrict__ p, double* partials,
                                                  unsigned* arrived, double* sc) {
    const size_t n = m.nIC;
    double v[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int c = blockIdx.x * VT + threadIdx.x; c < m.nIC; c += gridDim.x * VT) {
        const double V = m.vol[c];
        double d = V, xc[5], acc[5];
        for (int q = 0; q < 5; q++) {
            xc[q] = x[5 * (size_t)c + q];
            acc[q] = V * xc[q];
        }
        for (int k = 0; k < 6; k++) {
            const int e = m.accf[k * n + c];
            const int f = e >= 0 ? e : ~e;
            int o = c;
            double w = 0.0;
            if (f < m.nIF) {
                o = e >= 0 ? m.nbr[f] : m.own[f];
                w = coef[f];
                d += w;
                for (int q = 0; q < 5; q++) acc[q] += w * (xc[q] - x[5 * (size_t)o + q]);
            }
            nbh[k * n + c] = o;
            wgt[k * n + c] = w;
        }
        const double rd = rcp(d);
        vol[c] = V;
        rdiag[c] = rd;
        const double a[5] = {(double)ar[c], (double)au[3 * c], (double)au[3 * c + 1], (double)au[3 * c + 2], (double)ae[c]};
        for (int q = 0; q < 5; q++) {
            const double rv = a[q] - acc[q], zv = rv * rd;
            r[5 * (size_t)c + q] = rv;
            p[5 * (size_t)c + q] = zv;
            v[q] += rv * zv;
            v[5 + q] += rv * rv;
        }
    }
    double s[10];
    if (grid_sums<10>(v, partials, arrived, s))
        for (int q = 0; q < 5; q++) {
            sc[q] = s[q];
            sc[15 + q] = s[5 + q];
        }
}

// q = A p and alpha = r.z / p.q. The products are of differences, V p + sum w (p - p_nb): the shorter
// diagonal p - sum w p_nb rounds at the size of w p, which for a smooth field and strong diffusion is
// far above that of the result (200 cells in a row, w = 1e4 V: error of the solution 5.7e-14 against
// 3.0e-15, w = 1e6 V: 3.0e-12 against 3.2e-14).
__global__ void __launch_bounds__(VT) k_heat_apply(int n, const double* __restrict__ vol,
                                                   const double* __restrict__ wgt, const int* __restrict__ nbh,
                                                   const double* __restrict__ p, double* __restrict__ q,
                                                   double* partials, unsigned* arrived, double* sc) {
    double v[5] = {0, 0, 0, 0, 0};
    for (int c = blockIdx.x * VT + threadIdx.x; c < n; c += gridDim.x * VT) {
        const double V = vol[c];
        double pc[5], acc[5];
        for (int k = 0; k < 5; k++) {
            pc[k] = p[5 * (size_t)c + k];
            acc[k] = V * pc[k];
        }
        for (int s = 0; s < 6; s++) {
            const int o = nbh[(size_t)s * n + c];
            const double w = wgt[(size_t)s * n + c];
            for (int k = 0; k < 5; k++) acc[k] += w * (pc[k] - p[5 * (size_t)o + k]);
        }
        for (int k = 0; k < 5; k++) {
            q[5 * (size_t)c + k] = acc[k];
            v[k] += pc[k] * acc[k];
        }
    }
    double s[5];
    if (grid_sums<5>(v, partials, arrived, s))
        for (int k = 0; k < 5; k++) sc[5 + k] = s[k] != 0.0 ? sc[k] / s[k] : 0.0;
}

// x += alpha p, r -= alpha q; r.z, r.r and beta = r.z / (the r.z before)
__global__ void __launch_bounds__(VT) k_cg_update(int n, double* sc, const double* __restrict__ rdiag,
                                                  const double* __restrict__ p, const double* __restrict__ q,
                                                  double* __restrict__ x, double* __restrict__ r, double* partials,
                                                  unsigned* arrived) {
    double v[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    double alpha[5];
    for (int k = 0; k < 5; k++) alpha[k] = sc[5 + k];
    for (int c = blockIdx.x * VT + threadIdx.x; c < n; c += gridDim.x * VT) {
        const double rd = rdiag[c];
        for (int k = 0; k < 5; k++) {
            const size_t i = 5 * (size_t)c + k;
            x[i] += alpha[k] * p[i];
            const double rv = r[i] - alpha[k] * q[i];
            r[i] = rv;
            v[k] += rv * (rv * rd);
            v[5 + k] += rv * rv;
        }
    }
    double s[10];
    if (grid_sums<10>(v, partials, arrived, s))
        for (int k = 0; k < 5; k++) {
            sc[10 + k] = sc[k] != 0.0 ? s[k] / sc[k] : 0.0;
            sc[k] = s[k];
            sc[15 + k] = s[5 + k];
        }
}

// p = r / diagonal + beta p
__global__ void __launch_bounds__(VT) k_cg_direction(int n, const double* __restrict__ sc,
                                                     const double* __restrict__ rdiag, const double* __restrict__ r,
                                                     double* __restrict__ p) {
    const int c = blockIdx.x * VT + threadIdx.x;
    if (c >= n) return;
    const double rd = rdiag[c];
    for (int k = 0; k < 5; k++) {
        const size_t i = 5 * (size_t)c + k;
        p[i] = r[i] * rd + sc[10 + k] * p[i];
    }
}

template <typename R, typename S>
__global__ void __launch_bounds__(VT) k_heat_out(MeshDev<R> m, const double* __restrict__ x, S* __restrict__ ar,
                                                 S* __restrict__ au, S* __restrict__ ae) {
    const int c = blockIdx.x * VT + threadIdx.x;
    if (c >= m.nIC) return;
    const double V = m.vol[c];
    const double* y = x + 5 * (size_t)c;
    ar[c] = (S)(y[0] * V);
    for (int k = 0; k < 3; k++) au[3 * c + k] = (S)(y[1 + k] * V);
    ae[c] = (S)(y[4] * V);
}

}  // namespace

template <typename R, typename S>
int adjoint_viscosity_dev(Ctx* c, const S* rho, const S* rhoU, const S* rhoE, int kind, double scaling, double dt,
                          S* ar, S* au, S* ae, double* Mout, double* DTout, int* iters, cudaStream_t s) {
    const MeshDev<R>& m = meshOf<R>(c);
    const Phys& P = c->phys;
    const size_t n = c->nIC;
    auto blocks = [](size_t items) { return (int)((items + VT - 1) / VT); };
    // the kernels with sums run at most four blocks a SM, whose threads take several cells: a block's
    // share of the sums, and the last block's tail (which adds one partial a block), cost less
    const int nb = blocks(n), ns = std::min(nb, 4 * 152);
    if (!c->viscWork) {
        const size_t words = 2 * (size_t)c->nC + 2 * (size_t)c->nF + 4 * 5 * n + 2 * n + 6 * n + 10 * (size_t)nb + 64 + 3 * n;
        int st = ctx_alloc(c, (void**)&c->viscWork, sizeof(double) * words);
        if (st) return st;
    }
    double* sc = c->viscWork;                // 64 scalars: the CG's, the norm's factor, the arrival count
    double* fac = sc + 40;
    unsigned* arrived = (unsigned*)(sc + 48);
    // (every kernel leaves the arrival count zero, unless calls on this context overlapped)
    cudaError_t cleared = cudaMemsetAsync(arrived, 0, sizeof(unsigned), s);
    if (cleared != cudaSuccess) return cuda_fail(c, cleared, "adjoint viscosity work");
    double* M = sc + 64;                     // nC: the viscosity before its scaling (nIC values)
    double* snd = M + c->nC;                 // nC: sound speeds
    double* DT = snd + c->nC;                // nF
    double* coef = DT + c->nF;               // nF: dt A DT / delta
    double* x = coef + c->nF;                // four n x 5 vectors
    double* r = x + 5 * n;
    double* p = r + 5 * n;
    double* q = p + 5 * n;
    double* vol = q + 5 * n;
    double* rdiag = vol + n;
    double* wgt = rdiag + n;                 // 6 x n
    double* partials = wgt + 6 * n;          // 10 x nb
    int* nbh = (int*)(partials + 10 * (size_t)nb);   // 6 x n
    ProfScope ps(c, KID_ADJ_VISC, s);
    launch_prim<R, S>(c, rho, rhoU, rhoE, s);
    if (kind != AFVM_VISC_UNIFORM) k_visc_sound<R><<<blocks(c->nC), VT, 0, s>>>(m, P, (const R*)c->rec, snd);
    k_visc_cell<R><<<nb, VT, 0, s>>>(m, P, (const R*)c->rec, snd, kind, c->volTotal, scaling, M, partials, arrived, fac);
    k_visc_face<R><<<blocks(c->nF), VT, 0, s>>>(m, M, fac, dt, DT, coef);
    // PCG on (V + dt L) x = a, from x0 = a / V (the unsmoothed field per unit volume)
    k_heat_rhs<R, S><<<ns, VT, 0, s>>>(m, ar, au, ae, x, partials, arrived, sc);
    k_heat_init<R, S><<<ns, VT, 0, s>>>(m, coef, ar, au, ae, x, vol, rdiag, wgt, nbh, r, p, partials, arrived, sc);
    double hs[25];
    const int maxIt = 500, checkEvery = 4;
    int it = 0;
    for (;; it++) {
        if (it % checkEvery == 0 || it >= maxIt) {
            cudaError_t e = cudaMemcpyAsync(hs, sc, sizeof(double) * 25, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) return cuda_fail(c, e, "adjoint viscosity solve");
            bool done = true;
            for (int k = 0; k < 5; k++)
                if (!(hs[15 + k] <= 1e-26 * hs[20 + k])) done = false;
            if (done || it >= maxIt) break;
        }
        k_heat_apply<<<ns, VT, 0, s>>>(c->nIC, vol, wgt, nbh, p, q, partials, arrived, sc);
        k_cg_update<<<ns, VT, 0, s>>>(c->nIC, sc, rdiag, p, q, x, r, partials, arrived);
        k_cg_direction<<<nb, VT, 0, s>>>(c->nIC, sc, rdiag, r, p);
    }
    if (iters) *iters = it;
    k_heat_out<R, S><<<nb, VT, 0, s>>>(m, x, ar, au, ae);
    if (Mout) k_visc_scaled<R><<<blocks(c->nC), VT, 0, s>>>(m, M, fac, Mout);
    if (DTout) cudaMemcpyAsync(DTout, DT, sizeof(double) * c->nF, cudaMemcpyDeviceToDevice, s);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(c, e, "adjoint viscosity launch");
    if (it >= maxIt) return fail(c, AFVM_ERR_TIMEOUT, "adjoint viscosity: the heat equation did not converge");
    return AFVM_OK;
}

template int adjoint_viscosity_dev<double, double>(Ctx*, const double*, const double*, const double*, int, double,
                                                   double, double*, double*, double*, double*, double*, int*,
                                                   cudaStream_t);
template int adjoint_viscosity_dev<float, float>(Ctx*, const float*, const float*, const float*, int, double, double,
                                                 float*, float*, float*, double*, double*, int*, cudaStream_t);
template int adjoint_viscosity_dev<float, double>(Ctx*, const double*, const double*, const double*, int, double,
                                                  double, double*, double*, double*, double*, double*, int*,
                                                  cudaStream_t);

}  // namespace afvm
