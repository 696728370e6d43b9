// nk_transport.cuh — the face reconstructions of the thickness transport, shared by the forward stage
// (nk_coefficients.cu) and its reverse (nk_time_adjoint.cu).
#pragma once

#include "nk_kernels.cuh"

namespace nk {

// The face thickness that u H carries through a face (UpwindBiased(order = 1 or 3) and WENO(order = 5) of the
// reference's advection, restated from their published algorithms).  s[m + 2], m = -2..2, is the stage thickness m
// cells from the upwind cell s[2] of the face, m > 0 towards and past the face.  A periodic stencil wraps as often as
// the grid is short; a Bounded one takes the edge cell (the zero-gradient halo).
__device__ __forceinline__ int wide_map(int i, int n, int periodic) {
    if (periodic) { int r = i % n; return r < 0 ? r + n : r; }
    return i < 0 ? 0 : (i > n - 1 ? n - 1 : i);
}
__device__ __forceinline__ void stencil_x(const DevGrid<double>& g, const double* __restrict__ H, int f, int j, bool east, double* s) {
    int row = wide_map(j, g.Ny, g.py) * g.pitch;
#pragma unroll
    for (int m = -2; m <= 2; ++m) s[m + 2] = H[row + wide_map(east ? f - 1 + m : f - m, g.Nx, g.px)];
}
__device__ __forceinline__ void stencil_y(const DevGrid<double>& g, const double* __restrict__ H, int i, int f, bool north, double* s) {
    int col = wide_map(i, g.Nx, g.px);
#pragma unroll
    for (int m = -2; m <= 2; ++m) s[m + 2] = H[wide_map(north ? f - 1 + m : f - m, g.Ny, g.py) * g.pitch + col];
}
// WENO-5: the three third-order candidates, their Jiang-Shu smoothness indicators and the WENO-Z weights
// α_k = d_k (1 + τ / (β_k + ε)), τ = |β₀ - β₂|, ε = 1e-8, d = (1, 6, 3) / 10 (Jiang and Shu 1996; Borges et al. 2008,
// exponent 1).  Both reconstructions of one cell from s[m + 2] = its neighbours m = -2..2: `plus` at the face towards
// m > 0 and `minus` at the other.  The two share their indicators (mirrored: β₀ and β₂ change places), the weights'
// numerators over the common denominator Π(β_k + ε) and, over the product of the weights' sums, one division; the
// candidates are differences from the cell, so that all of it is 68 FP64 instructions a pair, 162 when each face's two
// reconstructions were evaluated by themselves.
__device__ __forceinline__ void weno5_cell(const double* s, double& plus, double& minus) {
    const double c = s[2];
    const double d1 = s[1] - s[0], d2 = c - s[1], d3 = s[3] - c, d4 = s[4] - s[3];
    const double D0 = d2 - d1, D1 = d3 - d2, D2 = d4 - d3;                       // second differences
    const double B0 = fma(2.0, d2, D0), B1 = d2 + d3, B2 = fma(-2.0, d3, D2);    // a - 4b + 3c, d - b, 3c - 4d + e
    const double eps = 1e-8, w13 = 13.0 / 12;
    const double e0 = fma(w13, D0 * D0, fma(0.25, B0 * B0, eps)), e1 = fma(w13, D1 * D1, fma(0.25, B1 * B1, eps)),
                 e2 = fma(w13, D2 * D2, fma(0.25, B2 * B2, eps));
    const double tau = fabs(e0 - e2);
    const double p0 = (e0 + tau) * (e1 * e2), p1 = (e1 + tau) * (e0 * e2), p2 = (e2 + tau) * (e0 * e1);
    const double p16 = 6 * p1, q0 = 3 * p0, q2 = 3 * p2;
    const double S = p0 + p16 + q2, M = p2 + p16 + q0;                           // the weights' sums, times 10
    const double g0 = fma(5.0, d2, -2.0 * d1), g1 = fma(2.0, d3, d2), g2 = fma(4.0, d3, -d4);   // 6 (candidate - c)
    const double h0 = fma(5.0, d3, -2.0 * d4), h1 = fma(2.0, d2, d3), h2 = fma(4.0, d2, -d1);   // 6 (c - candidate)
    const double r = (1.0 / 6) / (S * M);
    plus = fma(fma(p0, g0, fma(p16, g1, q2 * g2)) * M, r, c);
    minus = fma(-(fma(p2, h0, fma(p16, h1, q0 * h2)) * S), r, c);
}
__device__ __forceinline__ double weno5_face(const double* s) {
    double plus, minus;
    weno5_cell(s, plus, minus);
    return plus;
}
__device__ __forceinline__ double face_value(const ThicknessView& v, const double* s) {
    if (v.scheme == NK_ADVECTION_WENO) return weno5_face(s);
    return v.order == 3 ? (-s[1] + 5 * s[2] + 2 * s[3]) / 6 : s[2];
}


// ∂(face value)/∂s[m], m = 0..4, of the reconstructions above, for the reverse of the stage.  WENO-5 by the chain rule
// through its candidates qₖ, smoothness indicators βₖ and weights: with αₖ = dₖ (1 + τ / (βₖ + ε)), S = Σ αₖ and
// q = Σ αₖ qₖ / S, ∂q = Σ αₖ/S ∂qₖ + Σ bₖ ∂βₖ, where gₖ = dₖ (qₖ - q) / S gives b through ∂αₖ = dₖ (∂τ / (βₖ + ε) -
// τ ∂βₖ / (βₖ + ε)²) and ∂τ = sign(β₀ - β₂) (∂β₀ - ∂β₂).  Four divisions; a quotient for every term and neighbour took
// thirty-two.
__device__ __forceinline__ void weno5_face_gradient(const double* s, double* J) {
    const double a = s[0], b = s[1], c = s[2], d = s[3], e = s[4];
    const double sixth = 1.0 / 6;
    const double q0 = (2 * a - 7 * b + 11 * c) * sixth, q1 = (-b + 5 * c + 2 * d) * sixth, q2 = (2 * c + 5 * d - e) * sixth;
    const double A0 = a - 2 * b + c, B0 = a - 4 * b + 3 * c;
    const double A1 = b - 2 * c + d, B1 = b - d;
    const double A2 = c - 2 * d + e, B2 = 3 * c - 4 * d + e;
    const double b0 = 13.0 / 12 * A0 * A0 + 0.25 * B0 * B0, b1 = 13.0 / 12 * A1 * A1 + 0.25 * B1 * B1, b2 = 13.0 / 12 * A2 * A2 + 0.25 * B2 * B2;
    const double eps = 1e-8, r0 = 1 / (b0 + eps), r1 = 1 / (b1 + eps), r2 = 1 / (b2 + eps);
    const double tau = fabs(b0 - b2), sg = b0 >= b2 ? 1.0 : -1.0;
    const double a0 = 0.1 * (1 + tau * r0), a1 = 0.6 * (1 + tau * r1), a2 = 0.3 * (1 + tau * r2);
    const double rS = 1 / (a0 + a1 + a2), val = (a0 * q0 + a1 * q1 + a2 * q2) * rS;
    const double g0 = 0.1 * (q0 - val) * rS * r0, g1 = 0.6 * (q1 - val) * rS * r1, g2 = 0.3 * (q2 - val) * rS * r2;
    const double G = sg * (g0 + g1 + g2);
    const double c0 = G - tau * g0 * r0, c1 = -tau * g1 * r1, c2 = -G - tau * g2 * r2;   // ∂q/∂βₖ
    const double k13 = 13.0 / 6;
    const double u0 = c0 * k13 * A0, v0 = c0 * 0.5 * B0, u1 = c1 * k13 * A1, v1 = c1 * 0.5 * B1, u2 = c2 * k13 * A2, v2 = c2 * 0.5 * B2;
    const double w0 = a0 * rS * sixth, w1 = a1 * rS * sixth, w2 = a2 * rS * sixth;
    J[0] = 2 * w0 + u0 + v0;
    J[1] = -7 * w0 - w1 - 2 * u0 - 4 * v0 + u1 + v1;
    J[2] = 11 * w0 + 5 * w1 + 2 * w2 + u0 + 3 * v0 - 2 * u1 + u2 + 3 * v2;
    J[3] = 2 * w1 + 5 * w2 + u1 - v1 - 2 * u2 - 4 * v2;
    J[4] = -w2 + u2 + v2;
}
__device__ __forceinline__ void face_value_gradient(const ThicknessView& v, const double* s, double* J) {
    if (v.scheme == NK_ADVECTION_WENO) { weno5_face_gradient(s, J); return; }
    const double third[5] = {0, -1.0 / 6, 5.0 / 6, 2.0 / 6, 0}, first[5] = {0, 0, 1, 0, 0};
#pragma unroll
    for (int m = 0; m < 5; ++m) J[m] = v.order == 3 ? third[m] : first[m];
}

}  // namespace nk
