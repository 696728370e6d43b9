// nk_transfer.cuh — the index and weight rules of the multigrid transfers, shared by the grid-wide kernels
// (nk_multigrid.cu) and the coarse levels' cluster kernel (nk_cluster.cu).  Indices are 0-based: coarse point I gathers
// the fine points 2 I + a.
#pragma once

#include "nk_kernels.cuh"

namespace nk {

// ---- restriction / prolongation index rules (0-based) ------------------------------------------------------
__device__ __forceinline__ void offsets(bool face, int c, int& a0, int& a1) {
    if (c == 1) { a0 = 0; a1 = 0; } else if (face) { a0 = -1; a1 = 1; } else { a0 = -1; a1 = 2; }
}
__device__ __forceinline__ int wrapn(int i, int n) { int r = i % n; return r < 0 ? r + n : r; }
// restriction_index (multigrid_preconditioner.jl:268-271)
__device__ __forceinline__ int ridx(int I, int a, int Nf, bool periodic, bool face, int c) {
    if (c == 1) return I;
    int i = 2 * I + a;
    if (periodic) return wrapn(i, Nf);
    if (face) return i < 0 ? 0 : i;
    return i < 0 ? 0 : (i > Nf - 1 ? Nf - 1 : i);
}
// restriction_weight (:273-283)
template <typename T>
__device__ __forceinline__ T rweight(int I, int a, int Nc, bool periodic, bool face, int c) {
    if (c == 1) return T(1);
    if (face) {
        if (!periodic && 2 * I + a < 0) return T(0);
        return a == 0 ? T(1) : T(1) / T(2);
    }
    T w = (a == 0 || a == 1) ? T(3) / T(4) : T(1) / T(4);
    if (periodic) return w;
    bool outside = (I == 0 && a == -1) || (I == Nc - 1 && a == 2);
    bool folded = (I == 0 && a == 0) || (I == Nc - 1 && a == 1);
    w = w + (folded ? T(1) / T(4) : T(0));
    return outside ? T(0) : w;
}
// parents (:286-305)
template <typename T>
__device__ __forceinline__ void parents(int i, int Nc, bool periodic, bool face, int c, int& I1, int& I2, T& w1, T& w2) {
    if (c == 1) { I1 = i; I2 = i; w1 = T(1); w2 = T(0); return; }
    int I = i / 2;
    bool odd1 = (i % 2) == 0;   // the 1-based index i + 1 is odd
    if (face) {
        int up = periodic ? wrapn(I + 1, Nc) : I + 1;
        I1 = I; I2 = odd1 ? I : up;
        w1 = odd1 ? T(1) : T(1) / T(2);
        w2 = odd1 ? T(0) : T(1) / T(2);
    } else {
        int Ip = odd1 ? I - 1 : I + 1;
        I1 = I;
        I2 = periodic ? wrapn(Ip, Nc) : (Ip < 0 ? 0 : (Ip > Nc - 1 ? Nc - 1 : Ip));
        w1 = T(3) / T(4); w2 = T(1) / T(4);
    }
}

}  // namespace nk
