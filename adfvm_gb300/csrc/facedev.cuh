// Device-side loads of the face inputs from the cell records and the mesh tables.
#pragma once
#include "ctx.cuh"
#include "face.cuh"
#include "soft64.cuh"

namespace afvm {

// 16-byte vector loads of n values (n a multiple of 4 floats / 2 doubles; p 16-byte aligned)
__device__ __forceinline__ void load_vec(const double* __restrict__ p, double* o, int n) {
#pragma unroll
    for (int i = 0; i < n; i += 2) {
        double2 v = __ldg(reinterpret_cast<const double2*>(p + i));
        o[i] = v.x; o[i + 1] = v.y;
    }
}
__device__ __forceinline__ void load_vec(const float* __restrict__ p, float* o, int n) {
#pragma unroll
    for (int i = 0; i < n; i += 4) {
        float4 v = __ldg(reinterpret_cast<const float4*>(p + i));
        o[i] = v.x; o[i + 1] = v.y; o[i + 2] = v.z; o[i + 3] = v.w;
    }
}

// the geometry inputs of a face (what the VJP reads besides the tape). Q: the type the face
// physics computes with (R, or sd for FP64)
template <typename R, typename Q>
__device__ __forceinline__ void load_face_geometry(const MeshDev<R>& m, int f, FaceIn<Q>& in) {
    const size_t nF = m.nF;
    for (int k = 0; k < 3; k++) {
        in.N[k] = m.nrm[k * nF + f];
        in.D[k] = m.du[k * nF + f];
        in.qw0[k] = m.qw[k * nF + f];
        in.qw1[k] = m.qw[(3 + k) * nF + f];
    }
    in.lw0 = m.lw[f];
    in.lw1 = m.lw[nF + f];
    in.rdelta = m.rdlt[f];
    if constexpr (sizeof(R) == 8) {
        for (int k = 0; k < 3; k++) in.Nt[k] = m.ntd[k * nF + f];
        in.ND = m.ntd[3 * nF + f];
    } else {
        // FP32 face kernels are bound by their loads, not by their (FP32) arithmetic: formed here
        in.ND = dot3(in.N, in.D);
        for (int k = 0; k < 3; k++) in.Nt[k] = in.N[k] - in.ND * in.D[k];
    }
}

// a face's kind, its cells, and the cell whose gradient the neighbour side reads (a ghost's is a
// copy of its source's)
struct FaceAt {
    int kind, own, nbr, grad;
};
template <typename R>
__device__ __forceinline__ FaceAt face_at(const MeshDev<R>& m, int f) {
    FaceAt a;
    a.kind = f < m.nIF ? FACE_INTERNAL : (int)m.fkind[f - m.nIF];
    a.own = m.own[f];
    a.nbr = m.nbr[f];
    a.grad = f < m.nIF ? a.nbr : m.gsrc[a.nbr - m.nIC];
    return a;
}
// what a face reads of the mesh
template <typename R, typename Q>
__device__ __forceinline__ FaceAt load_face_mesh(const MeshDev<R>& m, int f, FaceIn<Q>& in) {
    const FaceAt a = face_at<R>(m, f);
    load_face_geometry<R, Q>(m, f, in);
    return a;
}

// the cell values of one face: primitives and gradients of both sides. most (for Q = sd): the
// largest magnitude seen among them (soft_seen); the mesh tables are checked when the context is
// made.
template <typename R, typename Q>
__device__ __forceinline__ void load_face_cells(const R* __restrict__ rec, const FaceAt& a, FaceIn<Q>& in,
                                                unsigned* most = nullptr) {
    R rP[REC], rN[REC], rNg[REC];
    load_vec(rec + (size_t)a.own * REC, rP, REC);
    load_vec(rec + (size_t)a.nbr * REC, rN, REC);
    if (a.grad == a.nbr) {
        for (int k = 0; k < REC; k++) rNg[k] = rN[k];
    } else {
        load_vec(rec + (size_t)a.grad * REC, rNg, REC);
    }
    if constexpr (!std::is_same<R, Q>::value)
        for (int k = 0; k < REC; k++) {
            soft_seen(*most, rP[k]);
            soft_seen(*most, k < R_GU ? rN[k] : rNg[k]);
        }
    for (int k = 0; k < 3; k++) { in.UP[k] = rP[k]; in.UN[k] = rN[k]; }
    in.TP = rP[R_T]; in.pP = rP[R_P];
    in.TN = rN[R_T]; in.pN = rN[R_P];
    for (int k = 0; k < 9; k++) { in.gUP[k] = rP[R_GU + k]; in.gUN[k] = rNg[R_GU + k]; }
    for (int k = 0; k < 3; k++) {
        in.gTP[k] = rP[R_GT + k]; in.gTN[k] = rNg[R_GT + k];
        in.gpP[k] = rP[R_GP + k]; in.gpN[k] = rNg[R_GP + k];
    }
}

// the 55 inputs of one face
template <typename R, typename Q>
__device__ __forceinline__ void load_face(const MeshDev<R>& m, const R* __restrict__ rec, int f, FaceIn<Q>& in,
                                          unsigned* most = nullptr) {
    load_face_cells<R, Q>(rec, load_face_mesh<R, Q>(m, f, in), in, most);
}

// soft_seen of a taped value; 1/eps of the entropy fix may be 1e30 (eps is at least `small`), in a
// uniform flow, and only meets eigenvalues below 2 eps
__device__ __forceinline__ void seen_taped(unsigned& most, int k, double x) {
    if (k != T_RE) soft_seen(most, x);
}

// a face's column of a device tape (value k of face f at tape[k nF + f]; p = tape + f)
template <typename R, typename Q = R>
struct TapeStore {
    R* p;
    size_t stride;
    __device__ __forceinline__ void put(int k, Q x) const { p[(size_t)k * stride] = raw(x); }
};
template <typename R, typename Q = R>
struct TapeLoad {
    static constexpr bool kFull = true;
    const R* p;
    size_t stride;
    unsigned* most = nullptr;      // as load_face
    __device__ __forceinline__ Q get(int k) const {
        const R x = __ldg(p + (size_t)k * stride);
        if constexpr (!std::is_same<R, Q>::value) seen_taped(*most, k, x);
        return x;
    }
};

}  // namespace afvm
