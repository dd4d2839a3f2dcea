// Discrete adjoint of one SSP-RK3 step with dt held fixed (the per-step VJP of the reference's
// adjoint sweep, apps/adjoint.py:101-126 and 268-291).
//
// Forward u0 -> u1 -> u2 -> u3 (timestep.py:27-55) is recomputed, then the three stages are
// reversed. For stage i with output adjoint abar_{i+1}, the residual seed is
// Rbar = -beta_ii dt abar_{i+1}, and J_R(u_i)^T Rbar is formed by three kernels, all gathers
// (no atomics, so every result is bitwise reproducible):
//   k_adj_flux   faces: Fbar = Rbar_P A/V_P - Rbar_N A/V_N, then the hand-derived face VJP
//                (face.cuh) -> a 40-value record per face (primitive/gradient adjoints of
//                both sides)
//   k_adj_cell1  cells: sum of the face records of the cell's 6 faces (its own side) and of the
//                gradient adjoints of the ghost cells it is the source of
//   k_adj_cell2  cells: transpose of the Green-Gauss gradient (own slots and, through the
//                back-slot weights, the neighbours'), ghost boundary conditions transposed,
//                objective gradient (stage 1), primitive VJP and the SSP-RK reverse update.
#include <cuda_runtime.h>
#include <cmath>
#include <type_traits>
#include "facedev.cuh"
#include "ff32.cuh"
#include "vane.cuh"

namespace afvm {

// face adjoint record, one side after the other: owner side [prims 5 | grads 15], then the
// neighbour (ghost) side [prims 5 | grads 15]
constexpr int FADJ = 40;
constexpr int CBAR = 20;   // per cell: primitive adjoint (5) then gradient adjoint (15)

// A face's adjoint record and forward values where the kernel keeps them.
// RowStage: the record as a row of 40 values, the forward values read from the tape column in
// global memory (or held in registers without a tape).
template <typename R>
struct RowStage {
    R* row;
    __device__ __forceinline__ void store(const R* v) const { stage_row<R, FADJ>(row, v); }
};
// ColumnStage: a column of shared memory of the thread's own (value k at col[k stride]) that
// holds the face's TAPE forward values - copied from the tape while the seeds are gathered, or
// written by the forward evaluation - and then, over them, the record.
template <typename R>
struct ColumnStage {
    R* col;
    static constexpr int stride = FLUX_BLOCK + 1;      // (odd: the copy-out reads rows)
    __device__ __forceinline__ void store(const R* v) const {
        for (int k = 0; k < FADJ; k++) col[k * stride] = v[k];
    }
    __device__ __forceinline__ void fetch(const R* __restrict__ tape, size_t nF) const {
        const unsigned dst = (unsigned)__cvta_generic_to_shared(col);
#pragma unroll
        for (int k = 0; k < TAPE; k++)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 8 * k * stride), "l"(tape + k * nF)
                         : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    __device__ __forceinline__ void fetched() const { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
};
// the forward values in a ColumnStage
template <typename R, typename Q>
struct TapeColumn {
    static constexpr bool kFull = true;
    R* p;
    unsigned* most;                // (TapeLoad)
    __device__ __forceinline__ void put(int k, Q x) const { p[k * ColumnStage<R>::stride] = raw(x); }
    __device__ __forceinline__ Q get(int k) const {
        const R x = p[k * ColumnStage<R>::stride];
        if constexpr (!std::is_same<R, Q>::value) seen_taped(*most, k, x);
        return x;
    }
};

// what a face's adjoint reads of the mesh
template <typename R, typename Q>
struct AdjFaceMesh {
    FaceAt at;
    FaceIn<Q> in;      // the geometry; the cell values where they are needed
    R wp, wn;          // A/V_L and, of an internal face, A/V_R
};
template <typename R, typename Q>
__device__ __forceinline__ void load_adj_face_at(const MeshDev<R>& m, int f, AdjFaceMesh<R, Q>& a) {
    a.at = face_at<R>(m, f);
    a.wp = m.wpf[f];
    a.wn = f < m.nIF ? m.wnf[f] : R(0);
}
template <typename R, typename Q>
__device__ __forceinline__ void load_adj_face_mesh(const MeshDev<R>& m, int f, AdjFaceMesh<R, Q>& a) {
    load_adj_face_at<R, Q>(m, f, a);
    load_face_geometry<R, Q>(m, f, a.in);
}

// the face flux's adjoint Fbar = coef (abar_P A/V_L - abar_N A/V_R), coef folded into the two weights
template <typename R, typename S, typename Q>
__device__ __forceinline__ void adj_seeds(const MeshDev<R>& m, const AdjFaceMesh<R, Q>& a, R coef,
                                          const S* __restrict__ ar, const S* __restrict__ au,
                                          const S* __restrict__ ae, int f, Q* Fb, unsigned* most = nullptr) {
    const int iP = a.at.own;
    Q wp = Q(coef) * Q(a.wp);
    R aP[5] = {R(ar[iP]), R(au[3 * iP]), R(au[3 * iP + 1]), R(au[3 * iP + 2]), R(ae[iP])};
    for (int k = 0; k < 5; k++) {
        if constexpr (!std::is_same<R, Q>::value) soft_seen(*most, aP[k]);
        Fb[k] = Q(aP[k]) * wp;
    }
    if (f < m.nIF) {
        const int iN = a.at.nbr;
        Q wn = Q(coef) * Q(a.wn);
        R aN[5] = {R(ar[iN]), R(au[3 * iN]), R(au[3 * iN + 1]), R(au[3 * iN + 2]), R(ae[iN])};
        for (int k = 0; k < 5; k++) {
            if constexpr (!std::is_same<R, Q>::value) soft_seen(*most, aN[k]);
            Fb[k] = Fb[k] - Q(aN[k]) * wn;
        }
    }
}

// one face's record of k_adj_flux into st; TAPED: the forward values of a non-boundary face come
// from its tape column instead of a re-evaluation of the face flux
template <typename R, typename S, bool TAPED, typename Q, typename Stage>
__device__ __forceinline__ void adj_face(const MeshDev<R>& m, const Phys& P, AdjFaceMesh<R, Q>& a,
                                         const R* __restrict__ rec, R coef, const S* __restrict__ ar,
                                         const S* __restrict__ au, const S* __restrict__ ae, int inviscid, int f,
                                         const Stage& st, const R* __restrict__ tape, unsigned* most = nullptr) {
    constexpr bool COLUMN = std::is_same<Stage, ColumnStage<R>>::value;
    const int kind = a.at.kind;
    const bool fromTape = TAPED && kind != FACE_BOUNDARY;
    if constexpr (TAPED && COLUMN)
        if (fromTape) st.fetch(tape + f, (size_t)m.nF);
    Q Fb[5];
    adj_seeds<R, S, Q>(m, a, coef, ar, au, ae, f, Fb, most);
    FaceIn<Q>& in = a.in;
    FaceBar<Q> b;
    zero_bar(b);
    if (fromTape) {
        if constexpr (COLUMN) {
            st.fetched();
            face_vjp_t<Q>(P, kind, inviscid != 0, in, TapeColumn<R, Q>{st.col, most}, Fb, b);
        } else {
            face_vjp_t<Q>(P, kind, inviscid != 0, in, TapeLoad<R, Q>{tape + f, (size_t)m.nF, most}, Fb, b);
        }
    } else {
        load_face_cells<R, Q>(rec, a.at, in, most);
        if constexpr (COLUMN && !TAPED) {
            if (kind != FACE_BOUNDARY) {
                // the forward's values through the column
                const TapeColumn<R, Q> t{st.col, most};
                Q F[5], maxaF;
                face_flux<Q>(P, kind, inviscid != 0, in, F, maxaF, t);
                face_vjp_t<Q>(P, kind, inviscid != 0, in, t, Fb, b);
            } else {
                face_vjp<Q>(P, kind, inviscid != 0, in, Fb, b);
            }
        } else {
            face_vjp<Q>(P, kind, inviscid != 0, in, Fb, b);
        }
    }
    const Q* src = &b.UP[0];
    R v[FADJ];
    for (int k = 0; k < 5; k++) { v[k] = raw(src[k]); v[20 + k] = raw(src[5 + k]); }
    for (int k = 0; k < 15; k++) { v[5 + k] = raw(src[10 + k]); v[25 + k] = raw(src[25 + k]); }
    st.store(v);
}

// the face again with the hardware's FP64 operations throughout (soft_flag)
template <typename R, typename S, bool TAPED>
__device__ __noinline__ void adj_face_again(const MeshDev<R>& m, const Phys& P, const R* rec, R coef, const S* ar,
                                            const S* au, const S* ae, int inviscid, int f, ColumnStage<R> st,
                                            const R* tape) {
    AdjFaceMesh<R, R> a;
    load_adj_face_mesh<R, R>(m, f, a);
    adj_face<R, S, TAPED, R>(m, P, a, rec, coef, ar, au, ae, inviscid, f, st, tape);
}

template <typename R, typename S, bool TAPED, int NT>
__global__ void __launch_bounds__(NT, 3 * FLUX_BLOCK / NT)
    k_adj_flux(MeshDev<R> m, Phys P, const R* __restrict__ rec, R coef, const S* __restrict__ ar,
               const S* __restrict__ au, const S* __restrict__ ae, R* __restrict__ fadj, int inviscid,
               const R* __restrict__ tape) {
    // the block's 40-value face records are staged here and written out contiguously: one
    // thread's 40 scalar stores at a 40-value stride would touch a new 32-byte sector each and
    // load L2 with eight partial writes per sector
    __shared__ __align__(16) R stage[NT * FADJ];
    const int f0 = blockIdx.x * NT;
    const int f = f0 + threadIdx.x;
    AdjFaceMesh<R, R> a;
    if (f < m.nF) load_adj_face_mesh<R, R>(m, f, a);
    dep_wait(rec, ar, au, ae, fadj, tape);
    if (f < m.nF)
        adj_face<R, S, TAPED, R>(m, P, a, rec, coef, ar, au, ae, inviscid, f, RowStage<R>{stage + threadIdx.x * FADJ},
                                 tape);
    __syncthreads();
    store_staged<R, FADJ, NT>(fadj, f0, min(NT, m.nF - f0), stage);
}

// FP32 and mixed contexts. The kernel waits for its loads (and issues 44 % of the time), so the
// warps a SM holds count: five blocks of 128. The geometry is loaded after the cells' values, when
// fewer registers are taken, and each warp copies its 32 records out by itself, in one bulk copy,
// without a barrier of the block: at 128^3 FP32 412 -> 375 us a launch, mixed 80^3 step and adjoint
// 1.160 -> 1.099 ms (six blocks spill, 498 us and 1.21 ms). All 61 forward values in
// shared memory, the Riemann part first, take 368 us at six blocks, but round differently: the
// operations and their order are those that FP32 results have always come from.
template <typename S, int NT>
__global__ void __launch_bounds__(NT, NT == 32 ? 12 : 5)
    k_adj_flux_f32(MeshDev<float> m, Phys P, const float* __restrict__ rec, float coef, const S* __restrict__ ar,
                   const S* __restrict__ au, const S* __restrict__ ae, float* __restrict__ fadj, int inviscid) {
    __shared__ __align__(16) float shared[NT / 32][32 * FADJ];
    const int lane = threadIdx.x & 31;
    const int f = blockIdx.x * NT + threadIdx.x;
    float* sh = shared[threadIdx.x >> 5];
    AdjFaceMesh<float, float> a;
    if (f < m.nF) load_adj_face_at<float, float>(m, f, a);
    dep_wait(rec, ar, au, ae, fadj);
    float v[FADJ];
    if (f < m.nF) {
        float Fb[5];
        adj_seeds<float, S, float>(m, a, coef, ar, au, ae, f, Fb);
        FaceIn<float>& in = a.in;
        FaceBar<float> b;
        zero_bar(b);
        load_face_geometry<float, float>(m, f, in);
        load_face_cells<float, float>(rec, a.at, in);
        // the VJP differentiates the absolute-form flux (the same function of the state as the
        // gauge form the forward evaluates)
        in.TP = rec_abs_T<float>(P, in.TP); in.TN = rec_abs_T<float>(P, in.TN);
        in.pP = rec_abs_p<float>(P, in.pP); in.pN = rec_abs_p<float>(P, in.pN);
        face_vjp<float, true>(P, a.at.kind, inviscid != 0, in, Fb, b);
        const float* src = &b.UP[0];
        for (int k = 0; k < 5; k++) { v[k] = src[k]; v[20 + k] = src[5 + k]; }
        for (int k = 0; k < 15; k++) { v[5 + k] = src[10 + k]; v[25 + k] = src[25 + k]; }
    }
    __syncwarp();
    if (f < m.nF) stage_row<float, FADJ>(sh + lane * FADJ, v);
    // the warp's records, contiguous in fadj, in one bulk copy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0 && f < m.nF) {
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(fadj + (size_t)f * FADJ),
                     "r"((unsigned)__cvta_generic_to_shared(sh)),
                     "r"((unsigned)(min(32, m.nF - f) * FADJ * sizeof(float)))
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
}

// The same with products, reciprocals and square roots on the integer pipes (soft64.cuh), FP64.
// Of 323 FP64 instructions a face of the taped VJP 233 are left: 3.71 -> 2.86 ms a launch of
// 6,340,608 faces (the FP64 pipe 84 % busy, 232 bytes a thread spilled at 168 registers; 2.3 ms when the
// pipe never waited). The forward values
// come through shared memory: read from global memory where they are used, the same kernel takes
// 3.05 ms at 168 registers and 3.07 ms at 128 (four blocks a SM). Untaped, the forward writes
// them there instead of holding 61 values in registers: 3 x 521 -> 3 x 310 us for 317,955
// faces (356 with the hardware's products).
constexpr size_t COLUMN_BYTES = sizeof(double) * TAPE * ColumnStage<double>::stride;
template <bool TAPED>
__global__ void __launch_bounds__(FLUX_BLOCK, 3)
    k_adj_flux_soft(const __grid_constant__ MeshDev<double> m, const __grid_constant__ Phys P,
                    const double* __restrict__ rec, double coef, const double* __restrict__ ar,
                    const double* __restrict__ au, const double* __restrict__ ae, double* __restrict__ fadj,
                    int inviscid, const double* __restrict__ tape) {
    extern __shared__ __align__(16) double columns[];
    constexpr int stride = ColumnStage<double>::stride;
    const int f0 = blockIdx.x * FLUX_BLOCK;
    const int f = f0 + threadIdx.x;
    AdjFaceMesh<double, sd> a;
    if (f < m.nF) load_adj_face_mesh<double, sd>(m, f, a);
    dep_wait(rec, ar, au, ae, fadj, tape);
    if (f < m.nF) {
        const ColumnStage<double> st{columns + threadIdx.x};
        soft_flag() = 0;
        unsigned most = 0;
        adj_face<double, double, TAPED, sd>(m, P, a, rec, coef, ar, au, ae, inviscid, f, st, tape, &most);
        if (__builtin_expect(most >= SOFT_LIMIT || soft_flag() != 0, 0))
            adj_face_again<double, double, TAPED>(m, P, rec, coef, ar, au, ae, inviscid, f, st, tape);
    }
    __syncthreads();
    // records i = j / 20 out of the columns, two values a step
    const int n = min(FLUX_BLOCK, m.nF - f0) * (FADJ / 2);
    double2* o = reinterpret_cast<double2*>(fadj + (size_t)f0 * FADJ);
    for (int j = threadIdx.x; j < n; j += FLUX_BLOCK) {
        const int i = j / (FADJ / 2), k = 2 * (j % (FADJ / 2));
        o[j] = make_double2(columns[k * stride + i], columns[(k + 1) * stride + i]);
    }
}

// the shared memory of k_adj_flux_soft on the context's device (before the first launch there)
int prepare_adjoint(Ctx* c) {
    cudaError_t e = cudaFuncSetAttribute(k_adj_flux_soft<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)COLUMN_BYTES);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_adj_flux_soft<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)COLUMN_BYTES);
    return e == cudaSuccess ? AFVM_OK : cuda_fail(c, e, "adjoint set-up");
}

// One cell's sum of its faces' adjoint records (and of the ghosts whose gradient is its own) in
// collate order. Bound by the records' bytes; a thread sums one 16-byte piece of its cell's record,
// so that the lanes side by side read a record's pieces side by side: with a thread a cell each
// load asked for 32 different lines. At 128^3 in FP32 246 -> 189 us (1.23 GB of records, indexes and
// results: 6.5 TB/s), at 64^3 in FP64 92 -> 62 us (320 and 640 threads a block: 63, 65).
constexpr int CELL1_BLOCK = 160;
template <typename R>
__global__ void __launch_bounds__(CELL1_BLOCK) k_adj_cell1(MeshDev<R> m, const R* __restrict__ fadj, R* __restrict__ cbar) {
    constexpr int PER = 16 / sizeof(R), PIECES = CBAR / PER;
    const long long t = blockIdx.x * (long long)CELL1_BLOCK + threadIdx.x;
    const int c = (int)(t / PIECES), k0 = PER * (int)(t % PIECES);
    int e[6], gs0 = 0, gs1 = 0;
    if (c < m.nIC) {
#pragma unroll
        for (int s = 0; s < 6; s++) e[s] = m.accf[s * (size_t)m.nIC + c];
        gs0 = m.gsStart[c];
        gs1 = m.gsStart[c + 1];
    }
    dep_wait(fadj, cbar);
    if (c >= m.nIC) return;
    R v[6][PER], acc[PER];
#pragma unroll
    for (int s = 0; s < 6; s++) {
        const bool ownerSide = e[s] >= 0;
        load_vec(fadj + (size_t)(ownerSide ? e[s] : ~e[s]) * FADJ + (ownerSide ? 0 : CBAR) + k0, v[s], PER);
    }
    // the first slot initialises the sums (adding it to zeros changes nothing but the sign of a
    // zero)
    for (int k = 0; k < PER; k++) acc[k] = v[0][k];
#pragma unroll
    for (int s = 1; s < 6; s++)
        for (int k = 0; k < PER; k++) acc[k] += v[s][k];
    // gradient adjoints of the ghosts whose gradient is a copy of this cell's
    for (int q = gs0; q < gs1; q++) {
        const R* r = fadj + (size_t)(m.nIF + m.gsList[q]) * FADJ + CBAR + k0;
        for (int k = 0; k < PER; k++)
            if (k0 + k >= 5) acc[k] += r[k];
    }
    stage_row<R, PER>(cbar + (size_t)c * CBAR + k0, acc);
}

// phiFbar_i = rv * sum_j G[i][j] sn_j  (transpose of grad += phiF (x) S N', scaled by 1/V)
template <typename R>
__device__ __forceinline__ void phi_bar(const R* G, const R* sn, R rv, R* pb) {
    for (int i = 0; i < 5; i++) pb[i] = rv * (G[3 * i] * sn[0] + G[3 * i + 1] * sn[1] + G[3 * i + 2] * sn[2]);
}

// p + a . b: in FP64, whose pipe binds the cell kernel, three FMAs onto p; the dot product by itself is
// a product, two FMAs and a sum (35 of the kernel's 205 FP64 instructions a cell: 786 -> 628 us a launch
// at 128^3, 119 -> 99 at 64^3). In FP32 the dot product first, as its results have always rounded.
template <typename R>
__device__ __forceinline__ R add_dot3(R p, const R* a, const R* b) {
    if constexpr (sizeof(R) == 8) return fma(a[2], b[2], fma(a[1], b[1], fma(a[0], b[0], p)));
    else return p + (a[0] * b[0] + a[1] * b[1] + a[2] * b[2]);
}

template <typename R, typename S, int STAGE, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 160 : BLOCK)
    k_adj_cell2(MeshDev<R> m, Phys P, const R* __restrict__ rec, const R* __restrict__ fadj,
                const R* __restrict__ cbar, const S* __restrict__ ur, const S* __restrict__ uu,
                const S* __restrict__ ue, const S* ainr, const S* ainu, const S* aine, S* a1r, S* a1u, S* a1e, S* a0r,
                S* a0u, S* a0e, S* sb, S* sr, S* su, S* se, double dt, int objective, int objStart, int objN,
                double obja, ff objaPair, VaneDev vane, const double* __restrict__ objSeed) {
    const CellAt<SPLIT> at;
    const int c = at.c;
    const bool first = !SPLIT || at.q0 == 0;        // the thread that goes on with the whole cell
    const size_t n = m.nIC;
    const size_t nF = m.nF;
    int nb[6], gs0 = 0, gs1 = 0;
    R bs[18], A[3];
    if (c < m.nIC) {
#pragma unroll
        for (int s = 0; s < 6; s++) nb[s] = m.gnb[s * n + c];
#pragma unroll
        for (int k = 0; k < 18; k++) bs[k] = m.gbs[k * n + c];
        for (int j = 0; j < 3; j++) A[j] = m.gAv[j * n + c];
        if (first) {
            gs0 = m.gsStart[c];
            gs1 = m.gsStart[c + 1];
        }
    }
    dep_wait(rec, fadj, cbar, ur, uu, ue, ainr, ainu, aine, a1r, a1u, a1e, a0r, a0u, a0e, sb, objSeed);
    R pbar[5];
    if constexpr (SPLIT) {
        __shared__ R sh[5 * 32];
        const int q = at.q0, lane = threadIdx.x & 31;
        if (c < m.nIC) {
            const R* r = cbar + (size_t)c * CBAR;
            R p = r[q], Gn[6][3];
            const R G[3] = {r[5 + 3 * q], r[6 + 3 * q], r[7 + 3 * q]};
#pragma unroll
            for (int s = 0; s < 6; s++)
                if (nb[s] < m.nIC)
                    for (int j = 0; j < 3; j++) Gn[s][j] = cbar[(size_t)nb[s] * CBAR + 5 + 3 * q + j];
            p = add_dot3(p, G, A);
#pragma unroll
            for (int s = 0; s < 6; s++)
                if (nb[s] < m.nIC) p = add_dot3(p, Gn[s], bs + 3 * s);
            sh[q * 32 + lane] = p;
        }
        __syncthreads();
        for (int i = 0; i < 5; i++) pbar[i] = sh[i * 32 + lane];
    } else {
        if (c >= m.nIC) return;
        // cell adjoint records in 16-byte loads (a record is 80 / 160 bytes, 16-byte aligned)
        R cb[CBAR];
        load_vec(cbar + (size_t)c * CBAR, cb, CBAR);
        for (int k = 0; k < 5; k++) pbar[k] = cb[k];
        const R* G = cb + 5;
        // the cell's own slots at once: sum_s (1 - w'_s) (G . S N'_s) / V = G . gAv
        for (int i = 0; i < 5; i++) pbar[i] = add_dot3(pbar[i], G + 3 * i, A);
#pragma unroll
        for (int s = 0; s < 6; s++) {
            if (nb[s] < m.nIC) {
                // neighbour's gradient: its slot for this face has S N'' = -S N' and weight gwb;
                // gbs_s = -gwb_s S N'_s / V_nb
                const R* b = bs + 3 * s;
                R cn[CBAR];
                load_vec(cbar + (size_t)nb[s] * CBAR, cn, CBAR);
                const R* Gn = cn + 5;
                for (int i = 0; i < 5; i++) pbar[i] = add_dot3(pbar[i], Gn + 3 * i, b);
            }
        }
    }
    // the state's adjoint of the stage's residual: J[0] and, of the others, J[k] jr
    S J[5], jr = S(0);
    auto whole_cell = [&]() {
        // ghost cells whose boundary value comes from this cell: transpose of the BC
        for (int q = gs0; q < gs1; q++) {
            int g = m.gsList[q];
            int f = m.nIF + g;
            int o = m.own[f];
            int s = m.gslot[g];
            R gp[5];
            const R* r = fadj + (size_t)f * FADJ;
            for (int k = 0; k < 5; k++) gp[k] = r[20 + k];
            R sn[3] = {m.gsn[(3 * s) * n + o], m.gsn[(3 * s + 1) * n + o], m.gsn[(3 * s + 2) * n + o]};
            R w = m.gw[s * n + o];
            R pb[5];
            phi_bar<R>(cbar + (size_t)o * CBAR + 5, sn, m.rvol[o], pb);
            for (int k = 0; k < 5; k++) gp[k] += w * pb[k];
            if (STAGE == 1 && objective == AFVM_OBJ_DRAG && f >= objStart && f < objStart + objN) {
                // drag = sum (p0 nx - mu(T0) (U0 - U0i)/delta) A, ghost values p0, T0, U0
                const R* rg = rec + (size_t)(m.nIC + g) * REC;
                const R* ro = rec + (size_t)o * REC;
                double T0 = rec_T<R>(P, rg[R_T]), U0 = rg[0], U0i = ro[0];
                double A = m.area[f], dl = m.dlt[f], nx = m.nrm[f];
                double mu = viscosity<double>(P, T0);
                double dmu = (P.muModel == AFVM_MU_SUTHERLAND) ? mu * (1.5 / T0 - 1.0 / (T0 + P.muTs)) : 0.0;
                gp[R_P] += (R)(obja * nx * A);
                gp[R_T] += (R)(-obja * dmu * (U0 - U0i) / dl * A);
                gp[0] += (R)(-obja * mu / dl * A);
            }
            if (STAGE == 1 && objSeed)
                for (int k = 0; k < 5; k++) gp[k] += (R)(obja * objSeed[(size_t)(m.nIC + g) * 5 + k]);
            int kind = m.gkind[g];
            int kU = kind & 7, kT = (kind >> 3) & 7, kp = (kind >> 6) & 7;
            if (kU == GK_TOTALPT) {
                // transpose of Ub = (U.d) d, Tb = Tt - (U.d)^2/(2 Cp), pb = pt (T/Tt)^kappa
                const R* rs = rec + (size_t)c * REC;      // this cell is the ghost's source (owner)
                R d[3] = {m.gval[g], m.gval[(size_t)m.nG + g], m.gval[2 * (size_t)m.nG + g]};
                R Tt = m.gval[3 * (size_t)m.nG + g], pt = m.gval[4 * (size_t)m.nG + g];
                R Un = rs[0] * d[0] + rs[1] * d[1] + rs[2] * d[2];
                R kap = consts<R>(P).ggm1;
                R Unb = dot3(gp, d) - gp[R_T] * Un / consts<R>(P).Cp;
                for (int k = 0; k < 3; k++) pbar[k] += Unb * d[k];
                pbar[R_T] += gp[R_P] * pt * kap * pow(rec_abs_T<R>(P, rs[R_T]) / Tt, kap - R(1)) / Tt;
                continue;
            }
            if (kU == GK_COPY) {
                for (int k = 0; k < 3; k++) pbar[k] += gp[k];
            } else if (kU == GK_SYM) {
                R nr[3] = {m.nrm[f], m.nrm[nF + f], m.nrm[2 * nF + f]};
                R un = dot3(gp, nr);
                for (int k = 0; k < 3; k++) pbar[k] += gp[k] - un * nr[k];
            }
            if (kT != GK_FIXED) pbar[R_T] += gp[R_T];
            if (kp != GK_FIXED) pbar[R_P] += gp[R_P];
        }
        // an objective evaluated by the caller: its gradient with respect to this cell's primitives
        if (STAGE == 1 && objSeed)
            for (int k = 0; k < 5; k++) pbar[k] += (R)(obja * objSeed[(size_t)c * 5 + k]);
        // objective on the stage-1 primitives
        if (STAGE == 1 && objective != AFVM_OBJ_NONE) {
            const R* rc = rec + (size_t)c * REC;
            bool done = false;
            if constexpr (sizeof(S) == 4)
                done = objective == AFVM_OBJ_KINETIC_ENERGY && kinetic_grad_ff(P.pair, objaPair, rc, m.vol[c], pbar);
            if (done) {
                // (added in pairs of floats)
            } else if (objective == AFVM_OBJ_KINETIC_ENERGY) {
                double U[3] = {rc[0], rc[1], rc[2]}, T = rec_T<R>(P, rc[R_T]), p = rec_p<R>(P, rc[R_P]), V = m.vol[c];
                double d = (P.Cv * T) * P.gm1;
                double rd = rcp(d);           // (Newton reciprocals: no IEEE divisions on the FP64 pipe)
                double rho = p * rd;
                double q = U[0] * U[0] + U[1] * U[1] + U[2] * U[2];
                for (int k = 0; k < 3; k++) pbar[k] += (R)(obja * rho * U[k] * V);
                pbar[R_P] += (R)(obja * 0.5 * q * V * rd);
                pbar[R_T] += (R)(-obja * 0.5 * q * V * rho * rcp(T));
            } else if (objective == AFVM_OBJ_SUM_T) {
                pbar[R_T] += (R)obja;
            } else if (objective == AFVM_OBJ_VANE) {
                int q = vane.cellPlane[c];
                if (q >= 0) {
                    double g5[5] = {0, 0, 0, 0, 0};
                    double U[3] = {rc[0], rc[1], rc[2]};
                    vane_cell_grad(P, vane, U, rec_T<R>(P, rc[R_T]), rec_p<R>(P, rc[R_P]), vane.planeArea[q], vane.sums[0],
                                   vane.sums[1], obja, g5);
                    for (int k = 0; k < 5; k++) pbar[k] += (R)g5[k];
                }
                if (vane.b != 0.0) {
                    for (int s = 0; s < 6; s++) {
                        int e = m.accf[s * n + c];
                        if (e < m.nIF) continue;          // owner-side boundary faces only
                        double k = vane.bHeatCoef[e - m.nIF];
                        if (k != 0.0) pbar[R_T] += (R)(-obja * vane.b * vane.rw2 * k);
                    }
                }
            } else if (objective == AFVM_OBJ_DRAG) {
                for (int s = 0; s < 6; s++) {
                    int e = m.accf[s * n + c];
                    if (e < objStart || e >= objStart + objN) continue;   // owner-side faces of the patch
                    const R* rg = rec + (size_t)m.nbr[e] * REC;
                    double T0 = rec_T<R>(P, rg[R_T]);
                    double mu = viscosity<double>(P, T0);
                    pbar[0] += (R)(obja * mu / (double)m.dlt[e] * (double)m.area[e]);
                }
            }
        }
        // primitive VJP (density.py:162-171)
        if constexpr (sizeof(S) == 4) {
            // float state: the density row without the low-Mach cancellation of the form below
            // (rhob and eb E/rho both hold pbar_p (g-1) E): with q = |U|^2/2 and e = E - q,
            //   J_rho = pbar_p (g-1) q - (pbar_U . U)/rho + (pbar_T/Cv) (q - e)/rho,
            // which float evaluates to its own rounding, so the FP32 context needs no FP64 here
            const PhysR<float>& Q = consts<float>(P);
            float rho = ur[c], rr = rcp(rho);
            float U[3] = {uu[3 * c] * rr, uu[3 * c + 1] * rr, uu[3 * c + 2] * rr};
            float E = ue[c] * rr;
            float q = 0.5f * (U[0] * U[0] + U[1] * U[1] + U[2] * U[2]);
            float e = E - q;
            float pT = pbar[R_T] * Q.rCv, pp = pbar[R_P] * Q.gm1;
            float eb = pT + pp * rho;
            for (int k = 0; k < 3; k++) J[1 + k] = pbar[k] - eb * U[k];
            J[4] = eb;
            jr = rr;
            J[0] = pp * q - (pbar[0] * U[0] + pbar[1] * U[1] + pbar[2] * U[2]) * rr + pT * (q - e) * rr;
        } else {
            double rho = ur[c], rU[3] = {uu[3 * c], uu[3 * c + 1], uu[3 * c + 2]}, rE = ue[c];
            double rr = rcp(rho);
            double U[3] = {rU[0] * rr, rU[1] * rr, rU[2] * rr};
            double E = rE * rr;
            double e = E - 0.5 * (U[0] * U[0] + U[1] * U[1] + U[2] * U[2]);
            double eb = (double)pbar[R_T] * P.rCv + (double)pbar[R_P] * P.gm1 * rho;
            double rhob = (double)pbar[R_P] * P.gm1 * e;
            double Ubt[3];
            for (int k = 0; k < 3; k++) Ubt[k] = (double)pbar[k] - eb * U[k];
            for (int k = 0; k < 3; k++) J[1 + k] = Ubt[k];
            J[4] = eb;
            jr = rr;
            J[0] = rhob - (Ubt[0] * U[0] + Ubt[1] * U[1] + Ubt[2] * U[2]) * rr - eb * E * rr;
        }
    };
    if constexpr (SPLIT) {
        __shared__ S shJ[6 * 32];
        const int lane = threadIdx.x & 31;
        if (first && c < m.nIC) {
            whole_cell();
            for (int q = 0; q < 5; q++) shJ[q * 32 + lane] = J[q];
            shJ[5 * 32 + lane] = jr;
        }
        __syncthreads();
        if (c >= m.nIC) return;
        J[0] = shJ[at.q0 * 32 + lane];
        jr = shJ[5 * 32 + lane];
    } else {
        whole_cell();
    }
    // SSP-RK reverse (timestep.py:35-45 transposed), in the state's type S. The source adjoint is
    // complete with stage 0, which writes it in the reference's layout (any part may be absent); the
    // stages before keep it in rows by component, as the outputs may alias inputs
    // (the roundings spelled out, the same in both forms of the kernel)
    auto plus_J = [&](S k, S x, int i, int q) {
        if (q == 0) return fma(k, x, J[i]);
        return fma(k, x, mul_rn(J[i], jr));
    };
#pragma unroll
    for (int i = 0; i < (SPLIT ? 1 : 5); i++) {
        const int q = SPLIT ? at.q0 : i;
        const S ain = state_at(ainr, ainu, aine, c, q);
        S& a0 = state_at(a0r, a0u, a0e, c, q);
        if (STAGE == 2) {
            sb[q * n + c] = S(2. / 3) * S(dt) * ain;
            a0 = S(1. / 3) * ain;
            state_at(a1r, a1u, a1e, c, q) = plus_J(S(2. / 3), ain, i, q);
        } else if (STAGE == 1) {
            sb[q * n + c] += S(1. / 4) * S(dt) * ain;
            a0 += S(3. / 4) * ain;
            state_at(a1r, a1u, a1e, c, q) = plus_J(S(1. / 4), ain, i, q);
        } else {
            const S src = sb[q * n + c] + S(dt) * ain;
            a0 += q == 0 ? ain + J[i] : fma(J[i], jr, ain);
            if (q == 0 ? sr != nullptr : (q == 4 ? se != nullptr : su != nullptr)) state_at(sr, su, se, c, q) = src;
        }
    }
}

template <typename R, typename S>
int adjoint_step_dev(Ctx* c, const S* rho, const S* rhoU, const S* rhoE, double dt, const S* Srho, const S* SrhoU,
                     const S* SrhoE, const S* rhoNa, const S* rhoUNa, const S* rhoENa, double obja, S* rhoa,
                     S* rhoUa, S* rhoEa, S* Srhoa, S* SrhoUa, S* SrhoEa, cudaStream_t s, const S* stages,
                     const R* tape, const ParamDev* params) {
    const MeshDev<R>& m = meshOf<R>(c);
    const Phys& P = c->phys;
    default_sources<S>(c, Srho, SrhoU, SrhoE);
    int inviscid = (P.muModel == AFVM_MU_CONSTANT && P.mu0 == 0.0) ? 1 : 0;
    S* u1[3] = {(S*)c->u1[0], (S*)c->u1[1], (S*)c->u1[2]};
    S* u2[3] = {(S*)c->u2[0], (S*)c->u2[1], (S*)c->u2[2]};
    const S* u0c[3] = {rho, rhoU, rhoE};
    const S* u1c[3] = {u1[0], u1[1], u1[2]};
    const S* u2c[3] = {u2[0], u2[1], u2[2]};
    // a tape holds the stage's cell records the primal step built (no primitive or gradient
    // launches here) and, in FP64, its face tape
    const R* faceTape = nullptr;
    const R* recTape = nullptr;
    split_tape<const R>(c, tape, faceTape, recTape);
    // the mesh gradients from face tapes; with nothing kept, from a whole step's
    bool byTape = false;
    const R* fluxes = nullptr;
    if constexpr (std::is_same<R, double>::value) {
        byTape = params && param_tapes(c, *params, faceTape, s);
        if (byTape && !stages && !tape && c->paramTapeWhole) fluxes = c->paramTape;
    }
    if (stages) {
        // the stage states the primal step kept (afvm_primal_step_stages)
        stage_views<S, const S>(stages, m.nIC, u1c, u2c);
    } else if (fluxes) {
        if constexpr (std::is_same<R, double>::value && std::is_same<S, double>::value) {
            R* t = c->paramTape + 3 * FREC * (size_t)m.nF;
            launch_forward_tape<R, S>(c, dt, u0c, u1, u2, Srho, SrhoU, SrhoE, t, c->paramTape, s);
            split_tape<const R>(c, t, faceTape, recTape);
        }
    } else {
        // forward recompute of the stage states
        launch_prim_grad<R, S>(c, rho, rhoU, rhoE, s);
        launch_flux_update<R, S>(c, 0, dt, nullptr, u0c, u1c, u2c, Srho, SrhoU, SrhoE, u1, s);
        launch_prim_grad<R, S>(c, u1[0], u1[1], u1[2], s);
        launch_flux_update<R, S>(c, 1, dt, nullptr, u0c, u1c, u2c, Srho, SrhoU, SrhoE, u2, s);
    }
    // reverse sweep
    S* A1[3] = {(S*)c->a1[0], (S*)c->a1[1], (S*)c->a1[2]};
    S* A2[3] = {(S*)c->a2[0], (S*)c->a2[1], (S*)c->a2[2]};
    R* fadj = (R*)c->fadj;
    R* cbar = (R*)c->cbar;
    S* sb = (S*)c->sbar;
    const Shape gF = shape_for(m.nF, FLUX_BLOCK), gC = shape_for(m.nIC, BLOCK);
    const bool split = split_cells(m.nIC);
    const double beta[3] = {1.0, 1. / 4, 2. / 3};
    for (int st = 2; st >= 0; st--) {
        const S* const* u = st == 0 ? u0c : (st == 1 ? u1c : u2c);
        const R* rec = recTape ? recTape + (size_t)st * m.nC * REC : (const R*)c->rec;
        if (!recTape) launch_prim_grad<R, S>(c, u[0], u[1], u[2], s);
        if (st == 1 && c->objective == AFVM_OBJ_VANE) launch_vane_sums<R>(c, s, nullptr, rec);
        // adjoint of this stage's output: a3 = seeds, a2 = A2, a1 = A1
        const S* ain[3];
        if (st == 2) { ain[0] = rhoNa; ain[1] = rhoUNa; ain[2] = rhoENa; }
        else if (st == 1) { ain[0] = A2[0]; ain[1] = A2[1]; ain[2] = A2[2]; }
        else { ain[0] = A1[0]; ain[1] = A1[1]; ain[2] = A1[2]; }
        R coef = (R)(-beta[st] * dt);
        const R* ft = faceTape ? faceTape + (size_t)st * TAPE * m.nF : nullptr;
        if constexpr (std::is_same<R, double>::value)
            if (byTape && !fluxes) {
                launch_flux<R>(c, false, rec, ft ? nullptr : c->paramTape, s);
                if (!ft) ft = c->paramTape;
            }
        {
            ProfScope ps(c, KID_ADJ_FLUX, s);
            const bool small = gF.threads == 32;
            if constexpr (std::is_same<R, float>::value) {
                launch_after(small ? k_adj_flux_f32<S, 32> : k_adj_flux_f32<S, FLUX_BLOCK>, gF.blocks, gF.threads, 0, s,
                             m, P, rec, coef, ain[0], ain[1], ain[2], fadj, inviscid);
            } else if (use_soft(c, m.nF) && std::fabs(coef) < 0x1p64) {
                launch_after(ft ? k_adj_flux_soft<true> : k_adj_flux_soft<false>, (m.nF + FLUX_BLOCK - 1) / FLUX_BLOCK,
                             FLUX_BLOCK, COLUMN_BYTES, s, m, P, rec, coef, ain[0], ain[1], ain[2], fadj, inviscid, ft);
            } else {
                auto flux = [&](auto taped, auto nt) {
                    launch_after(k_adj_flux<R, S, decltype(taped)::value, decltype(nt)::value>, gF.blocks, gF.threads,
                                 0, s, m, P, rec, coef, ain[0], ain[1], ain[2], fadj, inviscid, ft);
                };
                using Small = std::integral_constant<int, 32>;
                using Big = std::integral_constant<int, FLUX_BLOCK>;
                if (ft && small) flux(std::true_type{}, Small{});
                else if (ft) flux(std::true_type{}, Big{});
                else if (small) flux(std::false_type{}, Small{});
                else flux(std::false_type{}, Big{});
            }
        }
        {
            ProfScope ps(c, KID_ADJ_GATHER, s);
            const long long n = m.nIC * (CBAR * sizeof(R) / 16);
            launch_after(k_adj_cell1<R>, (int)((n + CELL1_BLOCK - 1) / CELL1_BLOCK), CELL1_BLOCK, 0, s, m, (const R*)fadj, cbar);
        }
        // the stage's share of the mesh / boundary-input gradients (before the cell kernel: the
        // adjoint outputs it writes may alias this stage's input adjoints)
        if constexpr (std::is_same<R, double>::value && std::is_same<S, double>::value)
            if (params) launch_param_grads<R, S>(c, *params, rec, coef, ain[0], ain[1], ain[2], st == 1, obja, s, byTape ? ft : nullptr,
                                             fluxes ? fluxes + (size_t)st * FREC * m.nF : (const R*)c->fflux);
        ProfScope ps(c, KID_ADJ_GRAD, s);
        S* const* a1 = st == 2 ? A2 : A1;      // (not written by the last stage)
        auto cells = [&](auto stage) {
            constexpr int ST = decltype(stage)::value;
            launch_after(split ? k_adj_cell2<R, S, ST, true> : k_adj_cell2<R, S, ST, false>,
                         split ? (m.nIC + 31) / 32 : gC.blocks, split ? 160 : gC.threads, 0, s, m, P, rec,
                         (const R*)fadj, (const R*)cbar, u[0], u[1], u[2], ain[0], ain[1], ain[2], a1[0], a1[1], a1[2],
                         rhoa, rhoUa, rhoEa, sb, Srhoa, SrhoUa, SrhoEa, dt, c->objective, c->objStart, c->objN, obja,
                         ff_of(obja), c->vane, c->objSeed);
        };
        if (st == 2) cells(std::integral_constant<int, 2>{});
        else if (st == 1) cells(std::integral_constant<int, 1>{});
        else cells(std::integral_constant<int, 0>{});
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(c, e, "adjoint step launch");
    return AFVM_OK;
}

#define AFVM_ADJ_INST(R, S)                                                                                    \
    template int adjoint_step_dev<R, S>(Ctx*, const S*, const S*, const S*, double, const S*, const S*, const S*, \
                                        const S*, const S*, const S*, double, S*, S*, S*, S*, S*, S*,             \
                                        cudaStream_t, const S*, const R*, const ParamDev*);
AFVM_ADJ_INST(double, double)
AFVM_ADJ_INST(float, float)
AFVM_ADJ_INST(float, double)

}  // namespace afvm
