// Primal residual and SSP-RK3 step on the device (sm_103a).
//
// One stage of the reference's time step (adFVM/timestep.py:27-55 over RCF.equation,
// adFVM/density.py:339-414) is four kernels:
//   k_prim    cells + ghost cells: conservative -> primitive (density.py:162-171) and the
//             ghost-cell boundary conditions (BCs.py via Solver.boundary, solver.py:106-114)
//   k_grad    cells: Green-Gauss gradient, a gather over the 6 cellFaces (op.py:45-63)
//   k_flux    faces: reconstruction, Riemann flux, viscous flux, CFL term (density.py:253-331)
//   k_update  cells: gather of the face fluxes in the reference's collate order (no atomics),
//             the SSP-RK stage combination (timestep.py:35-45) and, at stage 1, the CFL max
// Data: one record of REC values per cell (primitives + gradients), one FREC record per
// face, mesh constants in SoA arrays; the conservative state keeps the reference layout
// (rho (n), rhoU (n x 3), rhoE (n)).
#include <cuda_runtime.h>
#include "ctx.cuh"
#include "facedev.cuh"
#include "ff32.cuh"
#include "vane.cuh"

namespace afvm {

// RCF.primitive (adFVM/density.py:162-171) in double. One out-of-line body, so that a ghost
// cell and its source cell get bit-identical values.
__device__ __noinline__ void primitive_d(const Phys& P, double rho, double r0, double r1, double r2, double rhoE,
                                         double* out) {
    double rr = rcp(rho);
    double U0 = r0 * rr, U1 = r1 * rr, U2 = r2 * rr;
    double E = rhoE * rr;
    double e = E - 0.5 * (U0 * U0 + U1 * U1 + U2 * U2);
    out[0] = U0; out[1] = U1; out[2] = U2;
    out[4] = (P.gm1 * rho) * e;
    out[3] = e * P.rCv;
}

// FP32 state: velocity in float; the internal energy rho*e = rhoE - |rhoU|^2/(2 rho) (the low-Mach
// cancellation), the pressure and the temperature from the float state in pairs of floats, or in
// double where a value is out of their range
__device__ __noinline__ void primitive_f(const Phys& P, float rho, float r0, float r1, float r2,
                                         float rhoE, float* out) {
    float rr = rcp(rho);
    out[0] = r0 * rr; out[1] = r1 * rr; out[2] = r2 * rr;
    if (__builtin_expect(prim_ff(P.pair, rho, r0, r1, r2, rhoE, rr, out + R_P, out + R_T), 1)) return;
    double q = (double)r0 * r0 + (double)r1 * r1 + (double)r2 * r2;
    double rhoe = (double)rhoE - 0.5 * q * (double)rr;
    out[4] = (float)(P.gm1 * rhoe - P.gaugeP);
    out[3] = (float)(rhoe * (double)rr * P.rCv - P.gaugeT);
}

// primitives of one state (element type S) into the record type R
__device__ __forceinline__ void prim_values(const Phys& P, double r, double u0, double u1, double u2, double e,
                                            double* out) {
    primitive_d(P, r, u0, u1, u2, e, out);
}
__device__ __forceinline__ void prim_values(const Phys& P, float r, float u0, float u1, float u2, float e,
                                            float* out) {
    primitive_f(P, r, u0, u1, u2, e, out);
}
// FP64 state, FP32 record: the primitives in double, the gauge offsets of T and p taken in
// double, then rounded once
__device__ __forceinline__ void prim_values(const Phys& P, double r, double u0, double u1, double u2, double e,
                                            float* out) {
    double v[5];
    primitive_d(P, r, u0, u1, u2, e, v);
    v[3] -= P.gaugeT;
    v[4] -= P.gaugeP;
    for (int k = 0; k < 5; k++) out[k] = (float)v[k];
}

// primitives of cell c from the state arrays
template <typename R, typename S>
__device__ __forceinline__ void load_prim(const Phys& P, const S* rho, const S* rhoU, const S* rhoE, int c, R* out) {
    prim_values(P, rho[c], rhoU[3 * c], rhoU[3 * c + 1], rhoU[3 * c + 2], rhoE[c], out);
}

// the five primitives at the head of a 16-byte aligned record: a 16-byte store and a scalar
// (two L2 write requests a cell instead of five)
__device__ __forceinline__ void store_prims(float* r, const float* v) {
    *reinterpret_cast<float4*>(r) = make_float4(v[0], v[1], v[2], v[3]);
    r[4] = v[4];
}
__device__ __forceinline__ void store_prims(double* r, const double* v) {
    *reinterpret_cast<double2*>(r) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2*>(r + 2) = make_double2(v[2], v[3]);
    r[4] = v[4];
}

// one cell's term of a cell-sum objective on its primitives U (3), T, p (record values: FP32
// ones hold gauge offsets): AFVM_OBJ_KINETIC_ENERGY 0.5 rho |U|^2 V in the record type, or
// AFVM_OBJ_SUM_T the temperature; accumulated in double
template <typename R>
__device__ __forceinline__ double cell_objective(const Phys& P, int kind, const R* r, R vol) {
    if (kind == AFVM_OBJ_KINETIC_ENERGY) {
        R rho = rec_abs_p<R>(P, r[R_P]) * rcp((consts<R>(P).Cv * rec_abs_T<R>(P, r[R_T])) * consts<R>(P).gm1);
        return (double)(R(0.5) * rho * (r[0] * r[0] + r[1] * r[1] + r[2] * r[2]) * vol);
    }
    return rec_T<R>(P, r[R_T]);
}

// the objectives that are sums over cells (evaluated in the stage-0 update, which writes the
// objective stage's primitives)
inline bool cell_sum_objective(int kind) { return kind == AFVM_OBJ_KINETIC_ENERGY || kind == AFVM_OBJ_SUM_T; }

__device__ __forceinline__ double block_sum(double v, double* sh) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x < 32) {
        r = (threadIdx.x < blockDim.x / 32) ? sh[threadIdx.x] : 0.0;
        for (int off = 16; off > 0; off >>= 1) r += __shfl_down_sync(0xffffffffu, r, off);
    }
    return r;
}

// ghost cell g's primitives from its source cell's (v, replaced in place): the boundary
// conditions of BCs.py:62-184 (FP32 records: T and p as gauge offsets, so a zero-gradient
// ghost keeps its source's bits)
template <typename R>
__device__ __forceinline__ void ghost_prims(const MeshDev<R>& m, const Phys& P, int g, R* v) {
    int kind = m.gkind[g];
    int kU = kind & 7, kT = (kind >> 3) & 7, kp = (kind >> 6) & 7;
    const R gT = kGauge<R> ? consts<R>(P).gT : R(0), gP = kGauge<R> ? consts<R>(P).gP : R(0);
    if (kU == GK_TOTALPT) {
        // CBC_TOTAL_PT (BCs.py:178-184): Un = U.d, Ub = Un d, Tb = Tt - Un^2/(2 Cp),
        // pb = pt (T/Tt)^(gamma/(gamma-1)) with U, T of the owner cell
        R d[3] = {m.gval[g], m.gval[(size_t)m.nG + g], m.gval[2 * (size_t)m.nG + g]};
        R Tt = m.gval[3 * (size_t)m.nG + g], pt = m.gval[4 * (size_t)m.nG + g];
        R Un = dot3(v, d);
        R T = kGauge<R> ? v[3] + gT : v[3];
        for (int k = 0; k < 3; k++) v[k] = Un * d[k];
        v[3] = Tt - R(0.5) * Un * Un / consts<R>(P).Cp;
        v[4] = pt * pow(T / Tt, consts<R>(P).ggm1);
        if constexpr (kGauge<R>) {
            v[3] = v[3] - gT;
            v[4] = v[4] - gP;
        }
        return;
    }
    if (kU == GK_FIXED) {
        for (int k = 0; k < 3; k++) v[k] = m.gval[(size_t)k * m.nG + g];
    } else if (kU == GK_SYM) {
        int f = m.nIF + g;
        R n[3] = {m.nrm[f], m.nrm[(size_t)m.nF + f], m.nrm[2 * (size_t)m.nF + f]};
        R un = dot3(v, n);
        for (int k = 0; k < 3; k++) v[k] = v[k] - un * n[k];
    }
    if (kT == GK_FIXED) v[3] = kGauge<R> ? m.gval[3 * (size_t)m.nG + g] - gT : m.gval[3 * (size_t)m.nG + g];
    if (kp == GK_FIXED) v[4] = kGauge<R> ? m.gval[4 * (size_t)m.nG + g] - gP : m.gval[4 * (size_t)m.nG + g];
}

// dtcBits (may be NULL): the step's CFL maximum, cleared here
template <typename R, typename S>
__global__ void __launch_bounds__(BLOCK) k_prim(MeshDev<R> m, Phys P, const S* __restrict__ rho,
                                                const S* __restrict__ rhoU, const S* __restrict__ rhoE,
                                                R* __restrict__ rec, unsigned long long* dtcBits) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int g = t - m.nIC;
    const int src = g >= 0 && g < m.nG ? m.gsrc[g] : t;
    dep_wait(rho, rhoU, rhoE, rec);
    if (t == 0 && dtcBits) *dtcBits = 0;
    if (t < m.nIC) {
        R v[5];
        load_prim<R, S>(P, rho, rhoU, rhoE, t, v);
        store_prims(rec + (size_t)t * REC, v);
        return;
    }
    if (g >= m.nG) return;
    R v[5];
    load_prim<R, S>(P, rho, rhoU, rhoE, src, v);
    ghost_prims<R>(m, P, g, v);
    store_prims(rec + (size_t)t * REC, v);
}

// the mesh side of a cell's gradient: the neighbours and the mesh-only products of
//   sum_s phiF_s S N'_s / V with phiF_s = phi_c (1 - w'_s) + phi_nb w'_s, regrouped as
//   phi_c sum_s (1 - w'_s) S N'_s / V + sum_s phi_nb (w'_s S N'_s / V)
// (15 FMAs a slot; the face interpolation and the 1/V scaling were 25)
template <typename R>
struct GradSlots {
    int nb[6];
    R ws[18], a[3], cl[3];
};
template <typename R>
__device__ __forceinline__ void load_slots(const MeshDev<R>& m, int c, GradSlots<R>& g) {
    const size_t n = m.nIC;
#pragma unroll
    for (int s = 0; s < 6; s++) g.nb[s] = m.gnb[s * n + c];
#pragma unroll
    for (int k = 0; k < 18; k++) g.ws[k] = m.gws[k * n + c];
    for (int j = 0; j < 3; j++) g.a[j] = m.gAv[j * n + c];
    if constexpr (kGauge<R>)
        for (int j = 0; j < 3; j++) g.cl[j] = m.gcl[j * n + c];
}

template <typename R>
__device__ __forceinline__ void grad_cell(const Phys& P, const R* __restrict__ rec, int c, const GradSlots<R>& t,
                                          R* row) {
    // the five primitives of a record as one 16-byte load and a scalar (records are 16-byte
    // aligned)
    R phic[5];
    load_vec(rec + (size_t)c * REC, phic, 4);
    phic[4] = rec[(size_t)c * REC + 4];
    R g[15];
    for (int i = 0; i < 5; i++)
        for (int j = 0; j < 3; j++) g[3 * i + j] = phic[i] * t.a[j];
#pragma unroll
    for (int s = 0; s < 6; s++) {
        const R* ws = t.ws + 3 * s;
        R rn[5];
        load_vec(rec + (size_t)t.nb[s] * REC, rn, 4);
        rn[4] = rec[(size_t)t.nb[s] * REC + 4];
        for (int i = 0; i < 5; i++)
            for (int j = 0; j < 3; j++) g[3 * i + j] = g[3 * i + j] + rn[i] * ws[j];
    }
    if constexpr (kGauge<R>) {
        // FP32 records hold T - gT, p - gP: the gradient of the constant offsets is the offset
        // times the cell's sum of S N'/V, which warped faces leave nonzero
        for (int j = 0; j < 3; j++) {
            g[9 + j] = g[9 + j] + consts<R>(P).gT * t.cl[j];
            g[12 + j] = g[12 + j] + consts<R>(P).gP * t.cl[j];
        }
    }
    R v[REC];
    for (int k = 0; k < 5; k++) v[k] = phic[k];
    for (int k = 0; k < 15; k++) v[R_GU + k] = g[k];
    stage_row<R, REC>(row, v);
}

// the cell's whole record (its primitives again, then the gradients) is staged and the block's
// records written contiguously. Other blocks read the primitives of these records while they
// are rewritten: the rewrite stores the bits already there (each cell's primitives are read
// from its own record and written back unchanged), so every read sees the same value whether
// it lands before or after the store.
template <typename R, int NT>
__global__ void __launch_bounds__(NT) k_grad(MeshDev<R> m, Phys P, R* __restrict__ rec) {
    __shared__ __align__(16) R stage[NT * REC];
    const int c0 = blockIdx.x * NT;
    const int c = c0 + threadIdx.x;
    GradSlots<R> t;
    if (c < m.nIC) load_slots<R>(m, c, t);
    dep_wait(rec);
    if (c < m.nIC) grad_cell<R>(P, rec, c, t, stage + threadIdx.x * REC);
    __syncthreads();
    if (c0 < m.nIC) store_staged<R, REC, NT>(rec, c0, min(NT, m.nIC - c0), stage);
}

// the split form (CellAt): warp q of a block does component q of 32 cells
template <typename R>
__global__ void __launch_bounds__(160) k_grad_split(MeshDev<R> m, Phys P, R* __restrict__ rec) {
    __shared__ __align__(16) R stage[32 * REC];
    const CellAt<true> at;
    const int c = at.c, q = at.q0, c0 = blockIdx.x * 32;
    GradSlots<R> t;
    if (c < m.nIC) load_slots<R>(m, c, t);
    dep_wait(rec);
    if (c < m.nIC) {
        const R phi = rec[(size_t)c * REC + q];
        R g[3], nb[6];
#pragma unroll
        for (int s = 0; s < 6; s++) nb[s] = rec[(size_t)t.nb[s] * REC + q];
        for (int j = 0; j < 3; j++) g[j] = phi * t.a[j];
#pragma unroll
        for (int s = 0; s < 6; s++)
            for (int j = 0; j < 3; j++) g[j] = g[j] + nb[s] * t.ws[3 * s + j];
        if constexpr (kGauge<R>) {
            const R offset = q == R_T ? consts<R>(P).gT : consts<R>(P).gP;
            if (q >= R_T)
                for (int j = 0; j < 3; j++) g[j] = g[j] + offset * t.cl[j];
        }
        R* row = stage + (threadIdx.x & 31) * REC;
        row[q] = phi;
        for (int j = 0; j < 3; j++) row[R_GU + 3 * q + j] = g[j];
    }
    __syncthreads();
    if (c0 < m.nIC) store_staged<R, REC, 160>(rec, c0, min(32, m.nIC - c0), stage);
}

template <typename R>
static void launch_grad(Ctx* c, R* rec, cudaStream_t s) {
    const MeshDev<R>& m = meshOf<R>(c);
    ProfScope ps(c, KID_GRAD, s);
    const Shape g = shape_for(m.nIC, BLOCK);
    if (split_cells(m.nIC))
        launch_after(k_grad_split<R>, (m.nIC + 31) / 32, 160, 0, s, m, c->phys, rec);
    else
        launch_after(g.threads == 32 ? k_grad<R, 32> : k_grad<R, BLOCK>, g.blocks, g.threads, 0, s, m, c->phys, rec);
}


// TAPED: also writes the face tape (TAPE values a face, column-major: tape[k nF + f]) that
// k_adj_flux<..., true> reads back instead of re-evaluating the forward flux
// CFL: the stage whose CFL sum is taken (the second, density.py:405-413); the other stages
// store 0 in the CFL slot and skip its square root
// one face: Q is the type its physics computes with (R, or sd for FP64)
template <typename R, typename Q, bool TAPED, bool CFL>
__device__ __forceinline__ void flux_face(const MeshDev<R>& m, const Phys& P, const FaceAt& at, FaceIn<Q>& in,
                                          const R* __restrict__ rec, int f, R* __restrict__ fflux, int inviscid,
                                          R* __restrict__ tape, unsigned* most = nullptr) {
    const int kind = at.kind;
    load_face_cells<R, Q>(rec, at, in, most);
    Q F[5], maxaF;
    // (FP32 records hold gauge offsets and their fluxes are the gauge form; only FP64
    // contexts keep face tapes)
    if constexpr (TAPED && !kGauge<R>)
        face_flux<Q>(P, kind, inviscid != 0, in, F, maxaF, TapeStore<R, Q>{tape + f, (size_t)m.nF});
    else
        face_flux<Q, kGauge<R>>(P, kind, inviscid != 0, in, F, maxaF);
    R* out = fflux + (size_t)f * FREC;
    for (int k = 0; k < 5; k++) out[k] = raw(F[k]);
    out[5] = CFL ? raw(maxaF) : R(0);
}

// the face again with the hardware's FP64 operations throughout (soft_flag)
template <typename R, bool TAPED, bool CFL>
__device__ __noinline__ void flux_face_again(const MeshDev<R>& m, const Phys& P, const R* rec, int f, R* fflux,
                                             int inviscid, R* tape) {
    FaceIn<R> in;
    const FaceAt at = load_face_mesh<R, R>(m, f, in);
    flux_face<R, R, TAPED, CFL>(m, P, at, in, rec, f, fflux, inviscid, tape);
}

// SOFT (FP64): products, reciprocals and square roots on the integer pipes (soft64.cuh). The FP64
// pipe binds either form; of 298 FP64 instructions a face (52 DADD, 90 DMUL, 156 DFMA) 183 are
// left (50 DADD, 133 DFMA): 3.47 -> 2.33 ms a taped launch of 6,340,608 faces, 1.85 ms when the
// pipe never waited (it is 81 % busy: three warps a sub-partition, whose integer chains are
// serial; 168 registers spill about 300 bytes a thread into 376 of loads, 128 registers for four warps
// spill more than they hide, 2.42 ms, 255 for two 2.46).
template <typename R, bool TAPED, bool CFL, bool SOFT>
__global__ void __launch_bounds__(FLUX_BLOCK, sizeof(R) == 8 ? 3 : 8)
    k_flux(const __grid_constant__ MeshDev<R> m, const __grid_constant__ Phys P, const R* __restrict__ rec,
           R* __restrict__ fflux, int inviscid, R* __restrict__ tape) {
    // (the 6-value face records are stored directly: staging them through shared memory, as
    // the 20- and 40-value records are, made this kernel slower - 0.217 -> 0.269 ms at 128^3 in
    // FP32 - the barrier costs more than the six partly coalesced stores)
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    using Q = std::conditional_t<SOFT, sd, R>;
    FaceIn<Q> in;
    FaceAt at = {};
    if (f < m.nF) at = load_face_mesh<R, Q>(m, f, in);
    dep_wait(rec, fflux, tape);
    if (f >= m.nF) return;
    if constexpr (SOFT) {
        soft_flag() = 0;
        unsigned most = 0;
        flux_face<R, Q, TAPED, CFL>(m, P, at, in, rec, f, fflux, inviscid, tape, &most);
        if (__builtin_expect(most >= SOFT_LIMIT || soft_flag() != 0, 0))
            flux_face_again<R, TAPED, CFL>(m, P, rec, f, fflux, inviscid, tape);
    } else {
        flux_face<R, Q, TAPED, CFL>(m, P, at, in, rec, f, fflux, inviscid, tape);
    }
}

// a 6-value face flux record in three 8- (FP32) or 16-byte (FP64) loads; records start on
// multiples of 24 / 48 bytes
__device__ __forceinline__ void load_flux_record(const float* __restrict__ p, float* o) {
#pragma unroll
    for (int i = 0; i < FREC; i += 2) {
        float2 v = __ldg(reinterpret_cast<const float2*>(p + i));
        o[i] = v.x; o[i + 1] = v.y;
    }
}
__device__ __forceinline__ void load_flux_record(const double* __restrict__ p, double* o) {
#pragma unroll
    for (int i = 0; i < FREC; i += 2) {
        double2 v = __ldg(reinterpret_cast<const double2*>(p + i));
        o[i] = v.x; o[i + 1] = v.y;
    }
}

// reduce_max of the CFL sums (density.py:405-410): a warp's maximum, then an atomic one. Sums of
// magnitudes order like their bits, compared as integers (an FP64 comparison takes the FP64 pipe). A
// NaN wins every comparison, as in the reference's max (a NaN's bits are above every finite
// double's), so a state gone non-finite gives a non-finite CFL sum and the step reports it.
__device__ __forceinline__ void cfl_max(double d, unsigned long long* dtcBits) {
    unsigned long long b = (unsigned long long)__double_as_longlong(d);
    const unsigned hi = (unsigned)(b >> 32), top = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = __reduce_max_sync(0xffffffffu, hi == top ? (unsigned)b : 0u);
    if ((threadIdx.x & 31) == 0) atomicMax(dtcBits, ((unsigned long long)top << 32) | lo);
}

// StepEnd's work, by one block
__device__ __forceinline__ void step_end(const StepEnd& e) {
    __shared__ double sh[BLOCK / 32];
    double v = 0.0;
#pragma unroll 8
    for (int i = threadIdx.x; i < e.nPartials; i += blockDim.x) v += e.partials[i];
    const double s = block_sum(v, sh);
    if (threadIdx.x != 0) return;
    const double dtc = __longlong_as_double((long long)*e.dtcBits);
    *e.dtcBits = 0;
    if (e.objOut) *e.objOut = s;
    if (e.dtcOut) *e.dtcOut = dtc;
    if (e.host) {
        e.host[0] = dtc;
        if (e.objOut) e.host[1] = s;
    }
    if (e.dtNext) {
        const double d = *e.dt;
        if (e.dtHist) *e.dtHist = d;
        *e.dtNext = e.fixed ? d : fmin(2 * e.CFL / dtc, d * e.stepFactor);
    }
}

// Gather of the face fluxes (op.div / op.absDiv, op.py:12-29, collated in the order of
// density.py:390-402) and the SSP-RK3 stage update (timestep.py:35-45). SPLIT: the form of CellAt
// with a sixth warp for the CFL sum. SOFT (FP64, use_soft): the FP64 pipe binds; the gather's 30
// products of about 105 FP64 instructions a cell go to the integer pipes (soft64.cuh; the same bits),
// and four blocks a SM then hide their latency: 392 -> 304 us at 128^3, 171 -> 136 at 96^3, 62 -> 50 at
// 64^3 (two blocks 322, 143, 55; three 301, 136, 54); at 64 registers it spills 220
// to 290 bytes a thread. A cell with a flux of 2^64 or more gathers again with the hardware's.
template <typename R, typename S, int STAGE, bool SPLIT, bool SOFT>
__global__ void __launch_bounds__(SPLIT ? 192 : BLOCK, SOFT ? 4 : 0)
    k_update(MeshDev<R> m, const R* __restrict__ fflux, double dtv, const double* dtp, const S* u0r, const S* u0u,
             const S* u0e, const S* u1r, const S* u1u, const S* u1e, const S* u2r, const S* u2u, const S* u2e,
             const S* __restrict__ Sr, const S* __restrict__ Su, const S* __restrict__ Se, S* outr, S* outu, S* oute,
             unsigned long long* dtcBits, Phys P, R* __restrict__ recNext, int objKind,
             double* __restrict__ objPartials, StepEnd end) {
    // the gather (and the CFL sum) in the flux type R, the stage update in the state's type S:
    // under FP32 fluxes with an FP64 state the six fluxes are summed in FP32 (each carries FP32
    // rounding already; summing them in FP64 cost six FP64 conversions, products and sums a
    // cell and component) and the state is updated in FP64
    const size_t n = m.nIC;
    const CellAt<SPLIT> at;
    const int c = at.c;
    const bool first = !SPLIT || at.q0 == 0;        // the thread that goes on with the whole cell
    int e[6], gs0 = 0, gs1 = 0;
    R w[6];
    if (c < m.nIC) {
#pragma unroll
        for (int k = 0; k < 6; k++) {
            e[k] = m.accf[k * n + c];
            w[k] = m.accw[k * n + c];
        }
        if (first) {
            gs0 = m.gsStart[c];
            gs1 = m.gsStart[c + 1];
        }
    }
    dep_wait(fflux, dtp, u0r, u0u, u0e, u1r, u1u, u1e, u2r, u2u, u2e, Sr, Su, Se, recNext);
    if (STAGE == 2 && end.dtcBits && blockIdx.x == gridDim.x - 1) {
        step_end(end);
        return;
    }
    R dtc = R(0);
    S o[5];
    if (c < m.nIC) {
        // the sums start at -0, which the compiler drops from the first term's add (-0 + x is x,
        // while +0 + x is one more add; the values differ at most in the sign of a zero)
        R res[5] = {R(-0.0), R(-0.0), R(-0.0), R(-0.0), R(-0.0)};
        unsigned most = 0;
        auto gather = [&](auto soft) {
#pragma unroll
            for (int k = 0; k < 6; k++) {
                bool ownerSide = e[k] >= 0;
                int f = ownerSide ? e[k] : ~e[k];
                // the side's sign on the weight (one select a face, not one a term); each product
                // rounded before it is added, as the reference's collate sum does, so that equal
                // and opposite terms cancel exactly
                R ws = ownerSide ? w[k] : -w[k];
                if constexpr (SPLIT) {
                    const R F = fflux[(size_t)f * FREC + at.q0];
                    if (at.q0 == 5) dtc = dtc + F * w[k];
                    else res[1] = res[1] + mul_rn(F, ws);
                    // (the energy residual's gauge term takes the mass residual)
                    if (kGauge<R> && at.q0 == 4) res[0] = res[0] + mul_rn(fflux[(size_t)f * FREC], ws);
                } else {
                    R F[FREC];
                    load_flux_record(fflux + (size_t)f * FREC, F);
                    if constexpr (decltype(soft)::value) {
                        for (int q = 0; q < 5; q++) {
                            soft_seen(most, F[q]);
                            res[q] = res[q] + soft_mul(F[q], ws);
                        }
                    } else {
                        for (int q = 0; q < 5; q++) res[q] = res[q] + mul_rn(F[q], ws);
                    }
                    dtc = dtc + F[5] * w[k];
                }
            }
        };
        gather(std::integral_constant<bool, SOFT>{});
        if (SOFT && __builtin_expect(most >= SOFT_LIMIT, 0)) {
            for (int q = 0; q < 5; q++) res[q] = R(-0.0);
            dtc = R(0);
            gather(std::false_type{});
        }
        const S rdt = S(dtp ? *dtp : dtv);
#pragma unroll
        for (int i = 0; i < (SPLIT ? 1 : 5); i++) {
            const int q = SPLIT ? at.q0 : i;
            if (SPLIT && q == 5) break;
            S rs = S(res[SPLIT ? 1 : i]);
            // gauge-form fluxes (FP32): the energy residual is the gathered one plus gaugeH times
            // the mass residual, the momentum residual the gathered one plus gaugeP times the
            // cell's sum of A/V N (the gaugeP N the face fluxes leave out; zero when the cell's
            // face area vectors close), both added in the state's type
            if constexpr (kGauge<R>) {
                if (q == 4) rs = rs + S(P.gaugeH) * S(res[0]);
                // (a float state reads the float copy of the closure sums: half the bytes)
                if (q >= 1 && q <= 3)
                    rs = rs + S(P.gaugeP) * (sizeof(S) == 4 ? S(m.gcl[(q - 1) * n + c]) : S(m.gclD[(q - 1) * n + c]));
            }
            const S Sv = state_at(Sr, Su, Se, c, q), a = state_at(u0r, u0u, u0e, c, q);
            // u = sum_j alpha_j u_j - beta dt (R - S) with -beta dt formed once a cell
            S v;
            if (STAGE == 0) {
                const S k = -rdt;
                v = a + k * (rs - Sv);
            } else if (STAGE == 1) {
                const S b = state_at(u1r, u1u, u1e, c, q);
                const S k = S(-(1. / 4)) * rdt;
                v = (S(3. / 4) * a + S(1. / 4) * b) + k * (rs - Sv);
            } else {
                const S b = state_at(u2r, u2u, u2e, c, q);
                const S k = S(-(2. / 3)) * rdt;
                v = (S(1. / 3) * a + S(2. / 3) * b) + k * (rs - Sv);
            }
            o[i] = v;
            state_at(outr, outu, oute, c, q) = v;
        }
    }
    if constexpr (SPLIT) {
        __shared__ S sh[5 * 32];
        const int lane = threadIdx.x & 31;
        if (at.q0 < 5) sh[at.q0 * 32 + lane] = o[0];
        __syncthreads();
        if (STAGE == 1 && at.q0 == 5) {
            cfl_max(c < m.nIC ? (double)dtc : 0.0, dtcBits);
            return;
        }
        if (!first || !recNext) return;
        for (int q = 0; q < 5; q++) o[q] = sh[q * 32 + lane];
    }
    double objv = 0.0;     // this cell's term of a cell-sum objective (stage 0, objPartials)
    if (c < m.nIC && recNext) {
        // the next stage's k_prim, fused: this cell's primitives and those of the ghost
        // cells whose source it is, from the values just stored (the same bits k_prim
        // would read back)
        R v[5];
        prim_values(P, o[0], o[1], o[2], o[3], o[4], v);
        store_prims(recNext + (size_t)c * REC, v);
        if (STAGE == 0 && objPartials) objv = cell_objective<R>(P, objKind, v, m.vol[c]);
        for (int q = gs0; q < gs1; q++) {
            int g = m.gsList[q];
            R gv[5] = {v[0], v[1], v[2], v[3], v[4]};
            ghost_prims<R>(m, P, g, gv);
            store_prims(recNext + (size_t)(m.nIC + g) * REC, gv);
        }
    }
    if (STAGE == 0 && objPartials) {
        // the objective stage's primitives are the ones this stage-0 update writes: the
        // objective's block partial sums (the same terms and order as k_objective)
        if constexpr (SPLIT) {
            for (int off = 16; off > 0; off >>= 1) objv += __shfl_down_sync(0xffffffffu, objv, off);
            if (threadIdx.x == 0) objPartials[blockIdx.x] = objv;
        } else {
            __shared__ double osh[BLOCK / 32];
            double sum = block_sum(objv, osh);
            if (threadIdx.x == 0) objPartials[blockIdx.x] = sum;
        }
    }
    if (!SPLIT && STAGE == 1) cfl_max((double)dtc, dtcBits);
}

// rows of U (3), T, p with absolute T and p from records of stride `stride` (FP32 records hold
// gauge offsets) into out (n x 5)
template <typename R>
__global__ void __launch_bounds__(BLOCK) k_abs_prims(const R* __restrict__ rec, int stride, int n, Phys P,
                                                     R* __restrict__ out) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const R* r = rec + (size_t)t * stride;
    R* o = out + (size_t)t * 5;
    o[0] = r[0]; o[1] = r[1]; o[2] = r[2];
    o[3] = rec_abs_T<R>(P, r[3]);
    o[4] = rec_abs_p<R>(P, r[4]);
}
void launch_abs_prims(const Ctx* c, const float* rec, int stride, int n, float* out, cudaStream_t s) {
    if (n > 0) k_abs_prims<float><<<nblocks(n), BLOCK, 0, s>>>(rec, stride, n, c->phys, out);
}

// ---- objectives, evaluated on the ghost-completed primitives of stage 1 ----

// per-block partial sums; kinds: AFVM_OBJ_KINETIC_ENERGY, AFVM_OBJ_SUM_T (cells) and
// AFVM_OBJ_DRAG (faces [start, start+n) of one patch, templates/cylinder_test.py:9-19)
template <typename R>
__global__ void __launch_bounds__(BLOCK) k_objective(MeshDev<R> m, Phys P, const R* __restrict__ rec, int kind,
                                                     int start, int n, double* partials) {
    __shared__ double sh[BLOCK / 32];
    dep_wait(rec, partials);
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    double v = 0.0;
    if (t < n) {
        if (kind == AFVM_OBJ_KINETIC_ENERGY || kind == AFVM_OBJ_SUM_T) {
            // per-cell term in the working precision R, accumulated in double
            v = cell_objective<R>(P, kind, rec + (size_t)t * REC, m.vol[t]);
        } else {
            int f = start + t;
            const R* rN = rec + (size_t)m.nbr[f] * REC;
            const R* rP = rec + (size_t)m.own[f] * REC;
            double U0 = rN[0], U0i = rP[0], p0 = rec_p<R>(P, rN[R_P]), T0 = rec_T<R>(P, rN[R_T]);
            double nx = m.nrm[f];
            double mu = (P.muModel == AFVM_MU_SUTHERLAND) ? (P.muAs * (T0 * sqrt(T0))) / (T0 + P.muTs) : P.mu0;
            double mungUx = mu * (U0 - U0i) / (double)m.dlt[f];
            v = (p0 * nx - mungUx) * (double)m.area[f];
        }
    }
    double s = block_sum(v, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// turbine-vane objective on the stage-1 primitives (adFVM/objectives/vane.py:7-60): threads
// [0, nPlane) take the plane cells (pressure-loss and weighting terms), the next nHeat threads
// the heat-transfer faces; three block partial sums (FP64) in partials[0|1|2][block]
template <typename R>
__global__ void __launch_bounds__(BLOCK) k_obj_vane(MeshDev<R> m, Phys P, const R* __restrict__ rec, VaneDev v,
                                                    int nBlocks, double* partials) {
    __shared__ double sh0[BLOCK / 32], sh1[BLOCK / 32], sh2[BLOCK / 32];
    dep_wait(rec, partials);
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    double l = 0.0, w = 0.0, h = 0.0;
    if (t < v.nPlane) {
        const R* r = rec + (size_t)v.planeCells[t] * REC;
        double U[3] = {r[0], r[1], r[2]};
        vane_cell(P, v, U, rec_T<R>(P, r[R_T]), rec_p<R>(P, r[R_P]), v.planeArea[t], l, w);
    } else if (t < v.nPlane + v.nHeat) {
        int q = t - v.nPlane;
        int f = v.heatFaces[q];
        h = v.heatCoef[q] * (v.Tw - rec_T<R>(P, rec[(size_t)m.own[f] * REC + R_T]));
    }
    double s0 = block_sum(l, sh0), s1 = block_sum(w, sh1), s2 = block_sum(h, sh2);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = s0;
        partials[nBlocks + blockIdx.x] = s1;
        partials[2 * nBlocks + blockIdx.x] = s2;
    }
}

// fixed-order sums of the vane partials into sums[0..2]; with objOut, also the objective
// a L/W + b H/sum(A w)
__global__ void __launch_bounds__(BLOCK) k_vane_finish(const double* partials, int nBlocks, VaneDev v, double* sums,
                                                       double* objOut, double* objHost) {
    __shared__ double sh0[BLOCK / 32], sh1[BLOCK / 32], sh2[BLOCK / 32];
    dep_wait(partials);
    double a = 0.0, b = 0.0, c = 0.0;
    for (int i = threadIdx.x; i < nBlocks; i += BLOCK) {
        a += partials[i];
        b += partials[nBlocks + i];
        c += partials[2 * nBlocks + i];
    }
    double L = block_sum(a, sh0), W = block_sum(b, sh1), H = block_sum(c, sh2);
    if (threadIdx.x == 0) {
        sums[0] = L;
        sums[1] = W;
        sums[2] = H;
        const double J = v.a * (L / W) + v.b * (H * v.rw2);
        if (objOut) *objOut = J;
        if (objHost) *objHost = J;
    }
}

template <typename R>
void launch_vane_sums(Ctx* c, cudaStream_t s, double* objOut, const R* rec, double* objHost) {
    const MeshDev<R>& m = meshOf<R>(c);
    {
        ProfScope ps(c, KID_OBJECTIVE, s);
        launch_after(k_obj_vane<R>, c->nVaneBlocks, BLOCK, 0, s, m, c->phys, rec ? rec : (const R*)c->rec, c->vane,
                     c->nVaneBlocks, c->vanePartials);
    }
    ProfScope ps(c, KID_FINISH, s);
    launch_after(k_vane_finish, 1, BLOCK, 0, s, c->vanePartials, c->nVaneBlocks, c->vane, c->vaneSums, objOut,
                 objHost);
}

template <typename R, typename S>
void launch_prim(Ctx* c, const S* r, const S* ru, const S* re, cudaStream_t s, R* rec) {
    const MeshDev<R>& m = meshOf<R>(c);
    ProfScope ps(c, KID_PRIM, s);
    const Shape g = shape_for((long long)m.nIC + m.nG, BLOCK);
    launch_after(k_prim<R, S>, g.blocks, g.threads, 0, s, m, c->phys, r, ru, re, rec ? rec : (R*)c->rec, c->dtcBits);
}

template <typename R, typename S>
void launch_prim_grad(Ctx* c, const S* r, const S* ru, const S* re, cudaStream_t s, R* rec) {
    const MeshDev<R>& m = meshOf<R>(c);
    if (!rec) rec = (R*)c->rec;
    launch_prim<R, S>(c, r, ru, re, s, rec);
    launch_grad<R>(c, rec, s);
}

// the faces' fluxes (and their tape) from the cell records
template <typename R>
void launch_flux(Ctx* c, bool cfl, const R* rec, R* tape, cudaStream_t s) {
    const MeshDev<R>& m = meshOf<R>(c);
    const Phys& P = c->phys;
    R* ff = (R*)c->fflux;
    int inviscid = (P.muModel == AFVM_MU_CONSTANT && P.mu0 == 0.0) ? 1 : 0;
    ProfScope ps(c, KID_FLUX, s);
    const Shape g = shape_for(m.nF, FLUX_BLOCK);
    auto flux = [&](auto taped, auto withCfl, auto soft) {
        launch_after(k_flux<R, decltype(taped)::value, decltype(withCfl)::value, decltype(soft)::value>, g.blocks,
                     g.threads, 0, s, m, P, rec, ff, inviscid, tape);
    };
    auto by_cfl = [&](auto taped, auto soft) {
        if (cfl) flux(taped, std::true_type{}, soft);
        else flux(taped, std::false_type{}, soft);
    };
    if constexpr (sizeof(R) == 8) {
        const bool soft = use_soft(c, m.nF);
        if (tape && soft) by_cfl(std::true_type{}, std::true_type{});
        else if (tape) by_cfl(std::true_type{}, std::false_type{});
        else if (soft) by_cfl(std::false_type{}, std::true_type{});
        else by_cfl(std::false_type{}, std::false_type{});
    } else {
        by_cfl(std::false_type{}, std::false_type{});     // (FP32 contexts keep no face tape)
    }
}

// faces -> fluxes, then the gather + stage update u_{st+1} = ... (timestep.py:35-45)
template <typename R, typename S>
void launch_flux_update(Ctx* c, int st, double dt, const double* dtDev, const S* const* u0, const S* const* u1,
                        const S* const* u2, const S* Sr, const S* Su, const S* Se, S* const* out, cudaStream_t s,
                        bool nextPrims, R* tape, R* recIn, R* recOut, double* objPartials, const StepEnd* end) {
    const MeshDev<R>& m = meshOf<R>(c);
    const Phys& P = c->phys;
    R* rec = recIn ? recIn : (R*)c->rec;
    R* ff = (R*)c->fflux;
    launch_flux<R>(c, st == 1, rec, tape, s);
    const Shape g = shape_for(m.nIC, BLOCK);
    R* recNext = nextPrims ? (recOut ? recOut : rec) : nullptr;
    ProfScope ps(c, KID_UPDATE, s);
    const S* none = nullptr;
    const bool split = split_cells(m.nIC);
    const S *const *b = st == 1 ? u1 : u2, *b0 = st ? b[0] : none, *b1 = st ? b[1] : none, *b2 = st ? b[2] : none;
    auto update = [&](auto stage) {
        constexpr int ST = decltype(stage)::value;
        auto kernel = split ? k_update<R, S, ST, true, false> : k_update<R, S, ST, false, false>;
        if constexpr (sizeof(R) == 8)
            if (use_soft(c, m.nIC)) kernel = k_update<R, S, ST, false, true>;
        launch_after(kernel, (split ? (m.nIC + 31) / 32 : g.blocks) +
                     (ST == 2 && end ? 1 : 0), split ? 192 : g.threads, 0, s, m, ff, dt, dtDev, u0[0], u0[1], u0[2], b0,
                     b1, b2, b0, b1, b2, Sr, Su, Se, out[0], out[1], out[2], c->dtcBits, P, recNext, c->objective,
                     ST == 0 && recNext ? objPartials : nullptr, ST == 2 && end ? *end : StepEnd{});
    };
    if (st == 0) update(std::integral_constant<int, 0>{});
    else if (st == 1) update(std::integral_constant<int, 1>{});
    else update(std::integral_constant<int, 2>{});
}

template <typename S>
void default_sources(Ctx* c, const S*& Srho, const S*& SrhoU, const S*& SrhoE) {
    const S* zs = (const S*)c->zeroS;
    if (!Srho) Srho = zs;
    if (!SrhoU) SrhoU = zs + c->nIC;
    if (!SrhoE) SrhoE = zs + 4 * (size_t)c->nIC;
}

template <typename R, typename S>
int primal_step_dev(Ctx* c, const S* rho, const S* rhoU, const S* rhoE, double dt, const double* dtDev,
                    const S* Srho, const S* SrhoU, const S* SrhoE, S* rhoN, S* rhoUN, S* rhoEN,
                    double* dtcDev, double* objDev, cudaStream_t s, S* stages, R* tape, const StepEnd* rule,
                    bool primsReady, bool nextStep) {
    const MeshDev<R>& m = meshOf<R>(c);
    const Phys& P = c->phys;
    default_sources<S>(c, Srho, SrhoU, SrhoE);
    S* u1[3] = {(S*)c->u1[0], (S*)c->u1[1], (S*)c->u1[2]};
    S* u2[3] = {(S*)c->u2[0], (S*)c->u2[1], (S*)c->u2[2]};
    if (stages) stage_views<S, S>(stages, m.nIC, u1, u2);
    S* outN[3] = {rhoN, rhoUN, rhoEN};
    const S* u0c[3] = {rho, rhoU, rhoE};
    const S* u1c[3] = {u1[0], u1[1], u1[2]};
    const S* u2c[3] = {u2[0], u2[1], u2[2]};
    int nObjBlocks = 0;
    if (c->objective == AFVM_OBJ_VANE && !c->vaneSet)
        return fail(c, AFVM_ERR_BAD_ARG, "AFVM_OBJ_VANE needs afvm_set_objective_vane before the first step");
    // with a tape each stage's cell records are built in the tape's record part (kept for the
    // adjoint step), else in the context's one record buffer
    R* faceTape = nullptr;
    R* recTape = nullptr;
    split_tape<R>(c, tape, faceTape, recTape);
    R* recs[3];
    for (int st = 0; st < 3; st++) recs[st] = recTape ? recTape + (size_t)st * m.nC * REC : (R*)c->rec;
    for (int st = 0; st < 3; st++) {
        const S* const* in = st == 0 ? u0c : (st == 1 ? u1c : u2c);
        // the primitives of stages 1 and 2, and of a step that follows another in primal_run_dev,
        // were written by the update before
        if (st == 0 && !primsReady) launch_prim<R, S>(c, in[0], in[1], in[2], s, recs[0]);
        launch_grad<R>(c, recs[st], s);
        if (st == 1 && c->objSink) {
            // the objective stage's primitives U (3), T, p of every cell, ghosts included, for an
            // objective evaluated by the caller (absolute values: FP32 records add their gauge)
            if constexpr (kGauge<R>)
                k_abs_prims<R><<<nblocks(m.nC), BLOCK, 0, s>>>(recs[1], REC, m.nC, P, (R*)c->objSink);
            else
                cudaMemcpy2DAsync(c->objSink, 5 * sizeof(R), recs[1], REC * sizeof(R), 5 * sizeof(R), (size_t)m.nC,
                                  cudaMemcpyDeviceToDevice, s);
        }
        if (st == 1 && c->objective == AFVM_OBJ_VANE) {
            launch_vane_sums<R>(c, s, objDev, (const R*)recs[1], rule ? nullptr : c->hostOutDev + 1);
        } else if (st == 1 && c->objective != AFVM_OBJ_NONE) {
            int start = 0, n = m.nIC;
            if (c->objective == AFVM_OBJ_DRAG) { start = c->objStart; n = c->objN; }
            const Shape g = shape_for(n, BLOCK);
            nObjBlocks = cell_sum_objective(c->objective) && split_cells(n) ? (n + 31) / 32 : g.blocks;
            if (nObjBlocks > c->nPartials) return fail(c, AFVM_ERR_BAD_ARG, "objective partials overflow");
            // a cell-sum objective's partials were written by the stage-0 update
            if (n > 0 && !cell_sum_objective(c->objective)) {
                ProfScope ps(c, KID_OBJECTIVE, s);
                launch_after(k_objective<R>, nObjBlocks, g.threads, 0, s, m, P, (const R*)recs[1], c->objective, start,
                             n, c->partials);
            }
        }
        S* const* out = st == 0 ? u1 : (st == 1 ? u2 : outN);
        double* objPartials = (st == 0 && cell_sum_objective(c->objective) &&
                               shape_for(m.nIC, BLOCK).blocks <= c->nPartials)
                                  ? c->partials : nullptr;
        if (st == 0 && cell_sum_objective(c->objective) && !objPartials)
            return fail(c, AFVM_ERR_BAD_ARG, "objective partials overflow");
        StepEnd end = {};
        if (st == 2) {
            if (rule) end = *rule;
            end.partials = c->partials;
            end.nPartials = nObjBlocks;
            end.dtcBits = c->dtcBits;
            end.dtcOut = dtcDev;
            end.host = rule ? nullptr : c->hostOutDev;
            end.objOut = c->objective == AFVM_OBJ_VANE ? nullptr : objDev;    // (k_vane_finish's)
        }
        launch_flux_update<R, S>(c, st, dt, dtDev, u0c, u1c, u2c, Srho, SrhoU, SrhoE, out, s, st < 2 || nextStep,
                                 faceTape ? faceTape + (size_t)st * TAPE * m.nF : nullptr, recs[st],
                                 st < 2 ? recs[st + 1] : nullptr, objPartials, st == 2 ? &end : nullptr);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(c, e, "primal step launch");
    return AFVM_OK;
}

// a step's first two stages and the third's face flux again: its tape, the three stages' flux records
// (FREC values a face each) and the stage states u1, u2
template <typename R, typename S>
void launch_forward_tape(Ctx* c, double dt, const S* const* u0, S* const* u1, S* const* u2, const S* Srho,
                         const S* SrhoU, const S* SrhoE, R* tape, R* flux, cudaStream_t s) {
    const MeshDev<R>& m = meshOf<R>(c);
    R *face, *recs;
    split_tape<R>(c, tape, face, recs);
    const S *const u1c[3] = {u1[0], u1[1], u1[2]}, *const u2c[3] = {u2[0], u2[1], u2[2]};
    void* const own = c->fflux;
    launch_prim<R, S>(c, u0[0], u0[1], u0[2], s, recs);
    for (int st = 0; st < 3; st++) {
        R* rec = recs + (size_t)st * m.nC * REC;
        R* t = face + (size_t)st * TAPE * m.nF;
        c->fflux = flux + (size_t)st * FREC * m.nF;
        launch_grad<R>(c, rec, s);
        if (st == 2) launch_flux<R>(c, false, rec, t, s);
        else
            launch_flux_update<R, S>(c, st, dt, nullptr, u0, u1c, u2c, Srho, SrhoU, SrhoE, st == 0 ? u1 : u2, s, true,
                                     t, rec, rec + (size_t)m.nC * REC);
    }
    c->fflux = own;
}

template <typename R, typename S>
int primal_run_dev(Ctx* c, S* rho, S* rhoU, S* rhoE, int nSteps, double dt0, double CFL, double stepFactor,
                   int fixed, const S* Srho, const S* SrhoU, const S* SrhoE, double* dtHist, double* dtcHist,
                   double* objHist, cudaStream_t s) {
    // the step's dt and the next one's in turn; each step's last update writes the next step's
    // primitives as well
    double* dtDev[2] = {c->scal + 2, c->scal + 3};
    cudaMemcpyAsync(dtDev[0], &dt0, sizeof(double), cudaMemcpyHostToDevice, s);
    for (int n = 0; n < nSteps; n++) {
        StepEnd rule = {};
        rule.dt = dtDev[n & 1];
        rule.dtNext = dtDev[(n + 1) & 1];
        rule.dtHist = dtHist ? dtHist + n : nullptr;
        rule.CFL = CFL;
        rule.stepFactor = stepFactor;
        rule.fixed = fixed;
        int st = primal_step_dev<R, S>(c, rho, rhoU, rhoE, 0.0, dtDev[n & 1], Srho, SrhoU, SrhoE, rho, rhoU, rhoE,
                                    dtcHist ? dtcHist + n : c->scal, objHist ? objHist + n : c->scal + 1, s, nullptr,
                                    nullptr, &rule, n > 0, n + 1 < nSteps);
        if (st != AFVM_OK) return st;
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(c, e, "primal run launch");
    return AFVM_OK;
}

#define AFVM_PRIMAL_INST(R, S)                                                                                 \
    template int primal_step_dev<R, S>(Ctx*, const S*, const S*, const S*, double, const double*, const S*,       \
                                       const S*, const S*, S*, S*, S*, double*, double*, cudaStream_t, S*, R*,    \
                                       const StepEnd*, bool, bool);                                                 \
    template int primal_run_dev<R, S>(Ctx*, S*, S*, S*, int, double, double, double, int, const S*, const S*,     \
                                      const S*, double*, double*, double*, cudaStream_t);                         \
    template void launch_prim<R, S>(Ctx*, const S*, const S*, const S*, cudaStream_t, R*);                       \
    template void launch_prim_grad<R, S>(Ctx*, const S*, const S*, const S*, cudaStream_t, R*);                  \
    template void launch_flux_update<R, S>(Ctx*, int, double, const double*, const S* const*, const S* const*,   \
                                           const S* const*, const S*, const S*, const S*, S* const*, cudaStream_t,  \
                                           bool, R*, R*, R*, double*, const StepEnd*);
AFVM_PRIMAL_INST(double, double)
AFVM_PRIMAL_INST(float, float)
AFVM_PRIMAL_INST(float, double)
template void launch_flux<double>(Ctx*, bool, const double*, double*, cudaStream_t);
template void launch_forward_tape<double, double>(Ctx*, double, const double* const*, double* const*, double* const*,
                                                  const double*, const double*, const double*, double*, double*,
                                                  cudaStream_t);
template void default_sources<double>(Ctx*, const double*&, const double*&, const double*&);
template void default_sources<float>(Ctx*, const float*&, const float*&, const float*&);
template void launch_vane_sums<double>(Ctx*, cudaStream_t, double*, const double*, double*);
template void launch_vane_sums<float>(Ctx*, cudaStream_t, double*, const float*, double*);

}  // namespace afvm
