// nk_cg_cluster.cu — conjugate gradients on a small grid, the whole iteration in one thread-block cluster.
//
// The Jacobi-preconditioned (or unpreconditioned) step of conjugate_gradient.jl:209-220 is a few microseconds of FP64
// arithmetic on a grid of a few thousand cells, but its two grid-wide kernels with their device-wide sums take 16 us, most
// of it launch, index and load latency.  Here sixteen CTAs keep x, r, p, the coefficients and the preconditioner of their
// cells in registers for the whole solve, one cell a thread, and a step costs two cluster barriers.
//
// A step.  p lives in shared memory, masked, with a halo row from the CTAs above and below.  Every thread forms the two
// normal stresses and the corner shear of its cell (the products of Stage, nk_strip.cuh, so that the operator differences
// neighbours before it multiplies); the row of stresses below the CTA, the row of corners above it and the corners on a
// Bounded east wall are formed by the first threads.  p.q is summed over the cluster; x, r and z follow; z's edge rows go
// into the neighbours' halos by distributed shared memory under the barrier of the second sum, and the halo of p is
// advanced beside p itself.  Every CTA adds the sixteen partial sums in the same order, so all take the same decision.
//
// What binds it: the FP64 pipe (30 instructions a cell) and latency (two sums, two divisions and a square root a step).
// Measured, a Jacobi step with the two grid-wide kernels against this one: 16 x 16 16.8 -> 7.3 us, 84 x 40 16.6 -> 7.0,
// 128 x 64 16.8 -> 9.4; batches of 32: 64 x 32 34.5 -> 10.3, 84 x 40 48.4 -> 29.3, 128 x 64 81.0 -> 47.1.
#include <cooperative_groups.h>

#include "nk_kernels.cuh"

namespace nk {

namespace cg = cooperative_groups;

constexpr int CG_CLUSTER_CTAS = 16, CG_CLUSTER_THREADS = 512;

// Rows per CTA; 0 if the grid leaves a thread more than one cell (8192 cells on a grid of enough rows).  The limit is the
// register file, and at 8192 cells a step takes 9.4 us of which the sixteen SMs' FP64 pipes are busy for more than half:
// twice the cells would take as long as the grid-wide kernels' 17 us.
int cg_cluster_rows(int Nx, int Ny) {
    const int rows = (Ny + CG_CLUSTER_CTAS - 1) / CG_CLUSTER_CTAS;
    return (long long)rows * Nx <= CG_CLUSTER_THREADS ? rows : 0;
}
static size_t cg_cluster_smem(int Nx, int rows) {
    const size_t cells = (size_t)(rows + 2) * (Nx + 2);
    return cells * (sizeof(double2) + 3 * sizeof(double)) + 2 * (size_t)Nx * sizeof(double2) + (2 * (size_t)Nx + rows) * sizeof(double);
}

struct CGClusterSums {
    double part[2][CG_CLUSTER_THREADS];
    double cta[3][CG_CLUSTER_CTAS];   // the CTAs' sums: p.q, r.r, r.z
    double alpha, beta, rho, pq, rr, rnorm;
    int stop;
};

// The CTA's sum of part[w], by one warp and a fixed tree, into slot `which` of every CTA of the cluster.
__device__ __forceinline__ void cta_sum_to_cluster(cg::cluster_group& cl, CGClusterSums& S, int w, int which, int rank) {
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    double a[CG_CLUSTER_THREADS / 32];
#pragma unroll
    for (int k = 0; k < CG_CLUSTER_THREADS / 32; ++k) a[k] = k < nw ? S.part[w][lane + 32 * k] : 0.0;
#pragma unroll
    for (int h = CG_CLUSTER_THREADS / 64; h > 0; h >>= 1)
        if (nw > h) {
#pragma unroll
            for (int k = 0; k < h; ++k) a[k] += a[k + h];
        }
    const double t = warp_sum(a[0]);
    if (lane < (int)gridDim.x) *cl.map_shared_rank(&S.cta[which][rank], lane) = t;
}
__device__ __forceinline__ double cluster_total(const CGClusterSums& S, int which) {
    const int lane = threadIdx.x & 31;
    double t = lane < (int)gridDim.x ? S.cta[which][lane] : 0.0;
#pragma unroll
    for (int d = CG_CLUSTER_CTAS / 2; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
    return t;
}

template <bool UNI>
__global__ void __launch_bounds__(CG_CLUSTER_THREADS, 1) k_cg_cluster(CGView v, int rows) {
    NK_BATCH_ENTER(v.o.g, v)   // the same answer in every CTA of a cluster (one slot)
    SolverScalars* const sc = v.sc;
    if (read_done(sc)) return;
    cg::cluster_group cl = cg::this_cluster();
    const DevGrid<double>& g = v.o.g;
    const int Nx = g.Nx, Ny = g.Ny, W = Nx + 2, rank = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
    const int j0 = rank * rows, cnt = Ny - j0 < rows ? Ny - j0 : rows;   // at least one row
    const int warp = tid >> 5;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ CGClusterSums S;
    double2* const P = reinterpret_cast<double2*>(smem_raw);              // masked p, rows -1 .. cnt, columns -1 .. Nx
    double2* const Z = P + (rows + 2) * W;                                // masked z of the rows below and above
    double* const SX = reinterpret_cast<double*>(Z + 2 * Nx);
    double* const SY = SX + (rows + 2) * W;
    double* const T = SY + (rows + 2) * W;
    double* const ext = T + (rows + 2) * W;                               // coefficients of the stresses around the CTA
    // the rows below and above, and the CTAs that hold them (-1: beyond a Bounded edge)
    int js = j0 - 1, jn = j0 + cnt;
    if (js < 0 && g.py) js = Ny - 1;
    if (jn >= Ny) jn = g.py ? 0 : -1;
    const int south = js >= 0 ? js / rows : -1, north = jn >= 0 ? jn / rows : -1;

    const int jl = tid / Nx, i = tid - jl * Nx, j = j0 + jl, k = g.idx(i, j);
    const bool own = jl < cnt;
    const int q = own ? (jl + 1) * W + i + 1 : 0;
    const bool west = own && g.px && i == 0, east = own && g.px && i == Nx - 1;   // repeated in the pad columns
    double2 x = make_double2(0.0, 0.0), r = x, z = x, p = x, d = make_double2(1.0, 1.0);
    double eta = 0.0, cff = 0.0, cu = 0.0, cv = 0.0;
    unsigned m = U_INACTIVE | V_INACTIVE | U_IDENTITY | V_IDENTITY;
    const double h2 = g.h * g.h;
    auto masked = [](double2 a, unsigned f) { return make_double2((f & U_INACTIVE) ? 0.0 : a.x, (f & V_INACTIVE) ? 0.0 : a.y); };
    auto put = [&](double2 a) {
        P[q] = a;
        if (west) P[q + Nx] = a;
        if (east) P[q - Nx] = a;
    };
    auto put_halo = [&](int h, double2 a) {   // h: Nx columns below, Nx above
        const int c = h < Nx ? h : h - Nx;
        double2* row = P + (h < Nx ? 0 : (cnt + 1) * W) + 1;
        row[c] = a;
        if (g.px && c == 0) row[Nx] = a;
        if (g.px && c == Nx - 1) row[-1] = a;
    };
    for (int e = tid; e < (rows + 2) * W; e += nt) { P[e] = make_double2(0.0, 0.0); SX[e] = SY[e] = T[e] = 0.0; }
    __syncthreads();
    if (own) {
        const double4 c = v.o.coef[k];
        m = __ldg(v.o.mask + k);
        x = v.x[k];
        r = v.r[k];
        z = v.z[k];
        if (v.precond == NK_PRECONDITIONER_DIAGONAL) d = v.invd[k];
        eta = c.x;
        cff = (!g.px && i == 0) || (!g.py && j == 0) ? v.o.wall_factor * c.y : c.y;
        cu = (UNI ? h2 : g.dxf[i] * g.dyc[j]) * c.z;
        cv = (UNI ? h2 : g.dxc[i] * g.dyf[j]) * c.w;
        p = z;
        put(masked(p, m));
    }
    for (int h = tid; h < 2 * Nx; h += nt) {
        const int c = h < Nx ? h : h - Nx, row = h < Nx ? js : jn;
        double2 a = make_double2(0.0, 0.0);
        if (row >= 0) a = masked(v.z[g.idx(c, row)], __ldg(v.o.mask + g.idx(c, row)));
        put_halo(h, a);
        if (h < Nx) {
            ext[h] = js >= 0 ? v.o.coef[g.idx(c, js)].x : 0.0;
        } else {
            const double f = v.o.coef[g.idx(c, jn >= 0 ? jn : Ny)].y;
            ext[h] = jn < 0 || (!g.px && c == 0) ? v.o.wall_factor * f : f;
        }
    }
    if (!g.px)
        for (int h = tid; h < cnt; h += nt) ext[2 * Nx + h] = v.o.wall_factor * v.o.coef[g.idx(Nx, j0 + h)].y;
    const StopRule rule(sc);
    double rho = sc->rho;
    int it = sc->it, status = sc->status;
    cl.sync();
    for (;;) {
        // normal stresses and corner shear
        double sx = 0.0, sy = 0.0, t = 0.0;
        if (own) {
            const double2 e = P[q + 1], n = P[q + W], s = P[q - W], w = P[q - 1], c = masked(p, m);
            const double du = e.x - c.x, dv = n.y - c.y;
            if (UNI) {
                sx = eta * (2.0 * du + dv);
                sy = eta * (2.0 * dv + du);
                t = cff * ((c.x - s.x) + (c.y - w.y));
            } else {
                const double exx = du * g.rdxc[i], eyy = dv * g.rdyc[j], e2 = 2.0 * eta;
                sx = g.dyc[j] * (e2 * (2.0 * exx + eyy));
                sy = g.dxc[i] * (e2 * (2.0 * eyy + exx));
                t = cff * ((c.x - s.x) * g.rdyf[j] + (c.y - w.y) * g.rdxf[i]);
            }
            SX[q] = sx;
            SY[q] = sy;
            T[q] = t;
            if (east) SX[q - Nx] = sx;
            if (west) T[q + Nx] = t;
        }
        const int extra = 2 * Nx + (g.px ? 0 : cnt);
        for (int h = tid; h < extra; h += nt) {
            if (h < Nx) {   // the normal stress of the row below
                const double2 *c = P + h + 1;
                const double du = c[1].x - c[0].x, dv = c[W].y - c[0].y;
                if (UNI) SY[h + 1] = ext[h] * (2.0 * dv + du);
                else if (js >= 0) SY[h + 1] = g.dxc[h] * (2.0 * ext[h] * (2.0 * (dv * g.rdyc[js]) + du * g.rdxc[h]));
            } else {        // the corners of the row above and of the east wall
                const bool top = h < 2 * Nx;
                const int at = top ? (cnt + 1) * W + (h - Nx) + 1 : (h - 2 * Nx + 1) * W + Nx + 1;
                const double2 c = P[at];
                const double dy = c.x - P[at - W].x, dx = c.y - P[at - 1].y;
                if (UNI) T[at] = ext[h] * (dy + dx);
                else T[at] = ext[h] * (dy * g.rdyf[top ? j0 + cnt : j0 + h - 2 * Nx] + dx * g.rdxf[top ? h - Nx : Nx]);
            }
        }
        __syncthreads();
        double2 a = make_double2(0.0, 0.0);   // A p
        double pq = 0.0;
        if (own) {
            double du, dv;
            if (UNI) {
                du = 2.0 * (sx - SX[q - 1]) + (T[q + W] - t);
                dv = 2.0 * (sy - SY[q - W]) + (T[q + 1] - t);
            } else {
                du = (sx - SX[q - 1]) + g.dxf[i] * (T[q + W] - t);
                dv = (sy - SY[q - W]) + g.dyf[j] * (T[q + 1] - t);
            }
            a.x = (m & U_IDENTITY) ? p.x : cu * p.x - du;
            a.y = (m & V_IDENTITY) ? p.y : cv * p.y - dv;
            pq = fma(p.x, a.x, p.y * a.y);
        }
        S.part[0][tid] = pq;
        __syncthreads();
        if (warp == 0) cta_sum_to_cluster(cl, S, 0, 0, rank);
        cl.sync();
        if (warp == 0) {
            const double total = cluster_total(S, 0), alpha = total == 0.0 ? 0.0 : rho / total;
            if (tid == 0) { S.alpha = alpha; S.pq = total; }
        }
        __syncthreads();
        const double alpha = S.alpha;
        if (S.pq < 0.0 && status == NK_OK) status = NK_BREAKDOWN;
        double rr = 0.0, rz = 0.0;
        if (own) {
            x.x = x.x + alpha * p.x;
            x.y = x.y + alpha * p.y;
            r.x = r.x + (-alpha) * a.x;
            r.y = r.y + (-alpha) * a.y;
            z = v.precond == NK_PRECONDITIONER_DIAGONAL ? make_double2(r.x * d.x, r.y * d.y) : r;
            const double2 zm = masked(z, m);
            if (jl == 0 && south >= 0) cl.map_shared_rank(Z, south)[Nx + i] = zm;     // the row above the CTA below
            if (jl == cnt - 1 && north >= 0) cl.map_shared_rank(Z, north)[i] = zm;    // and below the CTA above
            rr = fma(r.x, r.x, r.y * r.y);
            rz = fma(r.x, z.x, r.y * z.y);
        }
        S.part[0][tid] = rr;
        S.part[1][tid] = rz;
        __syncthreads();
        ++it;
        if (nt > 32) {
            if (warp < 2) cta_sum_to_cluster(cl, S, warp, 1 + warp, rank);
        } else {
            cta_sum_to_cluster(cl, S, 0, 1, rank);
            cta_sum_to_cluster(cl, S, 1, 2, rank);
        }
        cl.sync();
        if (warp == 0) {   // beta
            const double total = cluster_total(S, 2), beta = rho == 0.0 ? 0.0 : total / rho;
            if (tid == 0) { S.beta = beta; S.rho = total; }
        }
        if (warp == 1 || nt == 32) {   // and beside it the stopping test
            const double total = cluster_total(S, 1), rn = sqrt(total);
            if ((tid & 31) == 0) { S.rr = total; S.rnorm = rn; S.stop = rule.stop(rn, it); }
        }
        __syncthreads();
        rho = S.rho;
        if (!finite_bits(S.rnorm)) status = NK_NONFINITE;
        if (S.stop) break;
        const double beta = S.beta;
        if (own) {
            p = make_double2(z.x + beta * p.x, z.y + beta * p.y);
            put(masked(p, m));
        }
        for (int h = tid; h < 2 * Nx; h += nt) {
            if ((h < Nx ? south : north) < 0) continue;
            const double2 b = Z[h], o = P[h < Nx ? h + 1 : (cnt + 1) * W + (h - Nx) + 1];
            put_halo(h, make_double2(b.x + beta * o.x, b.y + beta * o.y));
        }
        __syncthreads();
    }
    if (own) {
        v.x[k] = x;
        v.r[k] = r;
    }
    if (rank == 0 && tid == 0) {
        sc->pq = S.pq;
        sc->alpha = S.alpha;
        sc->beta = S.beta;
        sc->rho = S.rho;
        sc->rr = S.rr;
        sc->rnorm = S.rnorm;
        sc->it = it;
        sc->status = status;
        if (!rule.fixed && !(S.rnorm <= rule.tol)) sc->cg_unconverged += 1;
        sc->done = 1;
    }
    cl.sync();   // no CTA leaves while another may still write to its shared memory
}

void launch_cg_cluster(const CGView& v, cudaStream_t s) {
    const int Nx = v.o.g.Nx, Ny = v.o.g.Ny, rows = cg_cluster_rows(Nx, Ny);
    cudaLaunchConfig_t cfg = {};
    const int ctas = (Ny + rows - 1) / rows;
    cfg.gridDim = dim3(ctas, 1, batch_slots());
    cfg.blockDim = dim3((rows * Nx + 31) / 32 * 32);
    cfg.dynamicSmemBytes = cg_cluster_smem(Nx, rows);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (v.o.g.h != 0.0) cudaLaunchKernelEx(&cfg, k_cg_cluster<true>, v, rows);
    else cudaLaunchKernelEx(&cfg, k_cg_cluster<false>, v, rows);
    count_launch();
}
// Clusters above eight CTAs and the shared memory of the largest grid (one row of 512 cells a CTA) on the current device
// (never in a capture), and whether it has room for one.
bool cg_cluster_available() {
    const size_t smem = 96 * 1024;
    return cluster_can_be_placed(k_cg_cluster<true>, CG_CLUSTER_CTAS, CG_CLUSTER_THREADS, smem) &&
           cluster_can_be_placed(k_cg_cluster<false>, CG_CLUSTER_CTAS, CG_CLUSTER_THREADS, smem);
}

}  // namespace nk
