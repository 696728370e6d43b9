// nk_internal.cuh — shared device definitions of libnunatak_gb300.
//
// Device layout.  Every two-dimensional field of an Nx x Ny grid is stored in one pitched array of
// (Ny + 1) rows of `pitch` >= Nx + 1 elements, x fastest; element (i, j), 0-based, is
//   cell (i, j) for a Center-Center field, the west face of cell (i, j) for a Face-Center field,
//   the south face for a Center-Face field, the south-west corner for a Face-Face field.
// Index i = Nx holds the east wall face (Bounded x), row j = Ny the north wall face (Bounded y).
// A velocity vector stores (u, v) of the same (i, j) interleaved as one 16-byte (8-byte in FP32) pair,
// so one load brings both components of a cell; the coefficients of the operator are one packed record
// per (i, j): (eta_H at the centre, eta_H at the south-west corner, beta_u, beta_v).
//
// Halo semantics.  Oceananigans fills halos by a periodic wrap or, for cell-centred data in a Bounded
// direction, by copying the edge value.  The kernels read the same values through index maps: wrap()
// for Periodic directions, clamp() for Bounded ones.  Face data in a Bounded direction is never read
// unmasked outside 0..N, so clamping it is equivalent.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <type_traits>

#include "../../include/nunatak_gb300.h"

// Device context of the C ABI: the CUDA ordinal made current by every call, and the last error message.
struct nk_context {
    int device = 0;
    std::string error;
    cudaStream_t stream = nullptr;   // records the reference event
    cudaEvent_t ref = nullptr;       // time origin of nk_solve_stats::device_start_ms / device_end_ms
};

namespace nk {

constexpr int BX = 32;   // thread-block tile of the 2-D kernels: BX x BY cells
constexpr int BY = 8;
constexpr int BLOCK_THREADS = BX * BY;

// Mask bits of the operator (one byte per (i, j)).
constexpr uint8_t U_INACTIVE = 1;   // u point is a wall or ice free (and not prescribed): identity row, zero in strain rates
constexpr uint8_t V_INACTIVE = 2;
constexpr uint8_t U_WALL = 4;       // wall (peripheral) only: the viscosity masks walls, not ice-free points
constexpr uint8_t V_WALL = 8;
// Prescribed velocity (the Dirichlet extension; the reference has none): an identity row whose value, held fixed
// at the prescribed one, still enters the strain rates.  U_INACTIVE is cleared on such a face, so the reads of the
// strain rates test U_INACTIVE alone and the rows test U_IDENTITY.
constexpr uint8_t U_DIRICHLET = 16;
constexpr uint8_t V_DIRICHLET = 32;
constexpr uint8_t U_IDENTITY = U_INACTIVE | U_DIRICHLET;
constexpr uint8_t V_IDENTITY = V_INACTIVE | V_DIRICHLET;

template <typename T> struct Vec2;
template <> struct Vec2<double> { using type = double2; };
template <> struct Vec2<float> { using type = float2; };
template <typename T> struct Vec4;
template <> struct Vec4<double> { using type = double4; };
template <> struct Vec4<float> { using type = float4; };

// Grid of one multigrid level as the kernels see it.  Metric arrays hold indices -2 .. N+2 (the pointer
// is offset by 2): dxc(i) = cell width of centre i, dxf(i) = centre spacing at face i (west of centre i).
template <typename T>
struct DevGrid {
    int Nx, Ny, pitch;
    int px, py;                         // periodic flags
    const T* dxc; const T* dxf; const T* dyc; const T* dyf;      // spacings
    const T* rdxc; const T* rdxf; const T* rdyc; const T* rdyf;  // their reciprocals
    // A batched launch (gridDim.z slots of identical problems whose device arenas lie slot_stride bytes apart):
    // slot z of a block shifts every pointer by z * slot_stride and stops when its Picard flag p_done (slot 0's,
    // shifted the same way) is set.  Zero and null outside a batch.
    long long slot_stride = 0;
    const int* p_done = nullptr;
    // Every spacing of the level equal (dxc = dxf = dyc = dyf = h over the whole metric range, a regular square grid):
    // h, else 0.  The column-marching walk then takes the closed form of the stencil on such a grid.
    T h = T(0);

    __device__ __forceinline__ int idx(int i, int j) const { return j * pitch + i; }
    __device__ __forceinline__ static int wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }
    __device__ __forceinline__ static int clampi(int i, int lo, int hi) { return i < lo ? lo : (i > hi ? hi : i); }
    // index maps with halo semantics
    __device__ __forceinline__ int cx(int i) const { return px ? wrap(i, Nx) : clampi(i, 0, Nx - 1); }
    __device__ __forceinline__ int cy(int j) const { return py ? wrap(j, Ny) : clampi(j, 0, Ny - 1); }
    __device__ __forceinline__ int fx(int i) const { return px ? wrap(i, Nx) : clampi(i, 0, Nx); }
    __device__ __forceinline__ int fy(int j) const { return py ? wrap(j, Ny) : clampi(j, 0, Ny); }
    __device__ __forceinline__ int c_idx(int i, int j) const { return idx(cx(i), cy(j)); }   // Center-Center
    __device__ __forceinline__ int u_idx(int i, int j) const { return idx(fx(i), cy(j)); }   // Face-Center
    __device__ __forceinline__ int v_idx(int i, int j) const { return idx(cx(i), fy(j)); }   // Center-Face
    __device__ __forceinline__ int ff_idx(int i, int j) const { return idx(fx(i), fy(j)); }  // Face-Face
    // inactive_cell and peripheral_node (Oceananigans Grids/inactive_node.jl) for Bounded directions
    __device__ __forceinline__ bool out_x(int i) const { return !px && (i < 0 || i >= Nx); }
    __device__ __forceinline__ bool out_y(int j) const { return !py && (j < 0 || j >= Ny); }
    __device__ __forceinline__ bool peripheral_fc(int i, int j) const { return out_y(j) || out_x(i) || out_x(i - 1); }
    __device__ __forceinline__ bool peripheral_cf(int i, int j) const { return out_x(i) || out_y(j) || out_y(j - 1); }
    __device__ __forceinline__ bool peripheral_ff(int i, int j) const { return out_x(i) || out_x(i - 1) || out_y(j) || out_y(j - 1); }
    __device__ __forceinline__ T Az_fc(int i, int j) const { return dxf[i] * dyc[j]; }
    __device__ __forceinline__ T Az_cf(int i, int j) const { return dxc[i] * dyf[j]; }
    __device__ __forceinline__ T Az_cc(int i, int j) const { return dxc[i] * dyc[j]; }
};

// A velocity prescribed at the u face (i, j) / v face (i, j).  Prescribable faces are those of the solved rows,
// (i, j) in 0..Nx-1 x 0..Ny-1 (wrapped when periodic): the west and south boundary faces of a Bounded direction
// and every interior face, but not the east / north boundary faces, which no row of the operator solves.
__device__ __forceinline__ bool prescribed_u(const DevGrid<double>& g, const double2* ud, int i, int j) {
    if (!ud || (!g.px && (i < 0 || i >= g.Nx)) || (!g.py && (j < 0 || j >= g.Ny))) return false;
    return !isnan(ud[g.idx(g.px ? g.wrap(i, g.Nx) : i, g.py ? g.wrap(j, g.Ny) : j)].x);
}
__device__ __forceinline__ bool prescribed_v(const DevGrid<double>& g, const double2* ud, int i, int j) {
    if (!ud || (!g.px && (i < 0 || i >= g.Nx)) || (!g.py && (j < 0 || j >= g.Ny))) return false;
    return !isnan(ud[g.idx(g.px ? g.wrap(i, g.Nx) : i, g.py ? g.wrap(j, g.Ny) : j)].y);
}

// Per-solve scalars of conjugate gradients and Picard, device resident.
struct SolverScalars {
    double rho;          // r . z of the current step
    double alpha, beta;
    double pq;
    double rr;           // r . r
    double rz_old;       // r_new . z_old (flexible conjugate gradients)
    double r0, tol, rnorm;
    double picard_dd, picard_xx;   // ||x - x_prev||^2, ||x||^2
    double reltol, abstol;
    int it, done, status;
    int fixed, iterations, maxiter, flexible;
    unsigned int ticket;           // last-block counter of the fused reductions
    // Picard (picard.jl:63-90), evaluated on the device between the conjugate-gradient solves
    double p_reltol, p_abstol, p_D, p_X;
    int p_fixed, p_iterations, p_maxiter, p_it;
    int p_done, it_total, cg_unconverged;
    int r32_exp;                   // mixed precision: the FP32 residual in the V-cycle is r 2^-r32_exp, z = z32 2^r32_exp
    int r32_exp_next;              // exponent the next k_cg_update scales its residual with (from the latest ‖r‖)
};

// Binary exponent that brings a residual of norm `norm` near 1 before it is rounded to FP32.  Scaling by a power of
// two is exact, so the multigrid (linear and homogeneous from a zero guess) gives the same digits as unscaled,
// but right-hand sides of any magnitude stay clear of FP32 overflow and of its subnormal range.  Evaluated by
// one thread per kernel (it costs FP64 instructions); the cells apply it with scale_pow2.
__device__ __forceinline__ int residual_exponent(double norm) {
    const int ex = (int)(((unsigned)__double2hiint(norm) >> 20) & 0x7ffu);   // a norm carries no sign
    if (ex > 0 && ex < 0x7ff) return ex - 1023;   // a normal number, without FP64 instructions
    return (norm > 0.0 && isfinite(norm)) ? ilogb(norm) : 0;
}
__device__ __forceinline__ bool finite_bits(double x) { return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u; }

// x 2^k by an integer add to the exponent field (no FP64 instruction): exact for normal x and results.  Zeros,
// infinities and NaNs pass through; subnormal x and results below the normal range flush to a signed zero,
// results above it become infinite.
__device__ __forceinline__ double scale_pow2(double x, int k) {
    long long b = __double_as_longlong(x);
    int ex = (int)((b >> 52) & 0x7ff);
    if (ex == 0x7ff || k == 0) return x;
    long long sign = b & (long long)0x8000000000000000ULL;
    int en = ex + k;
    if (ex == 0 || en <= 0) return __longlong_as_double(sign);
    if (en >= 0x7ff) return __longlong_as_double(sign | 0x7ff0000000000000LL);
    return __longlong_as_double(b + ((long long)k << 52));
}

// f 2^k in FP64 on the integer units (an F2F conversion takes the FP64 pipe): exact, the bits of scale_pow2((double)f, k).
__device__ __forceinline__ double widen_pow2(float f, int k) {
    const unsigned u = __float_as_uint(f), a = u & 0x7fffffffu;
    const int ex = (int)(a >> 23), e = ex + 896 + k;   // 896 = 1023 - 127
    if (ex != 0 && ex != 255 && e > 0 && e < 2047)
        return __hiloint2double((int)((u & 0x80000000u) | ((a >> 3) + (unsigned)((896 + k) << 20))), (int)(a << 29));
    if (a == 0) return __hiloint2double((int)u, 0);
    return scale_pow2((double)f, k);
}
// (float)(x 2^k) on the integer units, rounded to nearest even: the bits of (float)scale_pow2(x, k)
__device__ __forceinline__ float narrow_pow2(double x, int k) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int ex = (int)((hi >> 20) & 0x7ffu), e = ex - 896 + k;
    if (ex != 0 && ex != 0x7ff && ex + k > 0 && ex + k < 0x7ff && e > 0 && e < 254) {
        const unsigned m = ((unsigned)e << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29), rest = lo & 0x1fffffffu;
        return __uint_as_float((hi & 0x80000000u) | (m + ((rest > 0x10000000u || (rest == 0x10000000u && (m & 1u))) ? 1u : 0u)));
    }
    return (float)scale_pow2(x, k);
}

// The sign of a flotation by its high word, on the integer units: a finite x >= +0, and a finite x < 0 of normal size.
// Neither holds for -0, subnormal negatives, infinities and NaN, which take the general expressions.
__device__ __forceinline__ bool surely_grounded(double x) { return (unsigned)__double2hiint(x) < 0x7ff00000u; }
__device__ __forceinline__ bool surely_floating(double x) {
    unsigned h = (unsigned)__double2hiint(x);
    return h >= 0x80100000u && h < 0xfff00000u;
}

// ---- warp / block reductions (fixed order, so results do not depend on scheduling) --------------------
template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums over a block of at most 256 threads of NV values (1 or 2); the results are valid in every thread.  One FP64
// instruction of a warp takes 64 cycles when nothing overlaps it and 19 of the SM's FP64 pipe otherwise, so the threads'
// values meet in shared memory and one warp per value adds them, a lane eight of them and then five shuffles: 8 dependent
// additions and 24 warp instructions for 256 threads and two values, where a butterfly in every warp takes 90.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV]) {
    const int tid = threadIdx.x + threadIdx.y * blockDim.x, lane = tid & 31, w = tid >> 5;
    const int nw = (blockDim.x * blockDim.y) >> 5;
    if (nw == 1) {
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] = warp_sum(v[q]);
        return;
    }
    __shared__ double sh[NV][256], res[NV];
    __syncthreads();   // a previous sum's results have been read
#pragma unroll
    for (int q = 0; q < NV; ++q) sh[q][tid] = v[q];
    __syncthreads();
    if (w < NV) {
        double a[8];   // by a tree: three dependent additions for eight warps
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = k < nw ? sh[w][lane + 32 * k] : 0.0;
        double t = nw <= 2 ? a[0] + a[1] : (nw <= 4 ? (a[0] + a[1]) + (a[2] + a[3]) : ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7])));
        t = warp_sum(t);
        if (lane == 0) res[w] = t;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = res[q];
}

// Deterministic grid-wide sums: every block writes its partial sums, the last block to arrive adds the partials in index
// order (fixed partition and tree) and returns true in all its threads with the totals in `v`.  `partials` holds one
// double2 per block.
template <int NV>
__device__ __forceinline__ bool grid_sum(double (&v)[NV], double2* partials, unsigned int* ticket) {
    static_assert(NV == 1 || NV == 2, "one or two values");
    __shared__ bool last;
    block_sum<NV>(v);
    const int nblocks = gridDim.x * gridDim.y, bid = blockIdx.x + blockIdx.y * gridDim.x;
    const int tid = threadIdx.x + threadIdx.y * blockDim.x, nt = blockDim.x * blockDim.y;
    if (tid == 0) {
        partials[bid] = make_double2(v[0], NV == 2 ? v[NV - 1] : 0.0);
        // releases this block's partials, acquires those of the blocks that came before
        unsigned int t;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(t) : "l"(ticket) : "memory");
        last = (t == (unsigned int)nblocks - 1);
    }
    __syncthreads();
    if (!last) return false;
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = 0.0;
    // k = tid, tid + nt, ... four at a time: the L2 reads (the partials of the other blocks are not in this SM's L1, so
    // __ldcg) are issued before their adds, and a fixed tree adds them
    for (int base = tid; base < nblocks; base += 4 * nt) {
        double2 p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            int k = base + u * nt;
            p[u] = k < nblocks ? __ldcg(&partials[k]) : make_double2(0.0, 0.0);
        }
        v[0] += (p[0].x + p[1].x) + (p[2].x + p[3].x);
        if (NV == 2) v[NV - 1] += (p[0].y + p[1].y) + (p[2].y + p[3].y);
    }
    block_sum<NV>(v);
    if (tid == 0) { *ticket = 0u; }
    return true;
}
__device__ __forceinline__ bool grid_sum2(double a, double b, double2* partials, unsigned int* ticket, double& ta, double& tb) {
    double v[2] = {a, b};
    bool last = grid_sum<2>(v, partials, ticket);
    ta = v[0];
    tb = v[1];
    return last;
}

// ---- batched launches ------------------------------------------------------------------------------------
// `p` moved by d bytes (null stays null): the same buffer in another slot of a batch.  Q is a pointer type,
// restrict-qualified or not (anything else fails the casts).
template <typename Q>
__device__ __forceinline__ void shift_ptr(Q& p, long long d) {
    if (p) p = reinterpret_cast<Q>(reinterpret_cast<unsigned long long>(p) + (unsigned long long)d);
}
template <typename T>
__device__ __forceinline__ void rebase(DevGrid<T>& g, long long d) {
    shift_ptr(g.dxc, d); shift_ptr(g.dxf, d); shift_ptr(g.dyc, d); shift_ptr(g.dyf, d);
    shift_ptr(g.rdxc, d); shift_ptr(g.rdxf, d); shift_ptr(g.rdyc, d); shift_ptr(g.rdyf, d);
    shift_ptr(g.p_done, d);
}
template <typename Q>
__device__ __forceinline__ void rebase(Q& p, long long d) { shift_ptr(p, d); }   // a pointer (restrict-qualified or not)
// The byte shift of this block's slot; false when the slot has stopped (its Picard flag is set).
template <typename T>
__device__ __forceinline__ bool batch_slot(const DevGrid<T>& g, long long& d) {
    d = 0;
    if (!g.slot_stride) return true;
    d = (long long)blockIdx.z * g.slot_stride;
    const int* pd = g.p_done;
    shift_ptr(pd, d);
    return !*(volatile const int*)pd;
}
inline __device__ void rebase_all(long long) {}
template <typename A, typename... Rest>
__device__ __forceinline__ void rebase_all(long long d, A& a, Rest&... rest) {
    rebase(a, d);
    rebase_all(d, rest...);
}
// First statement of every kernel of the solve: under a batched launch, stop for a finished slot and move the
// listed views and pointers (G's grid first) to this block's slot.
#define NK_BATCH_ENTER(G, ...)                                              \
    {                                                                       \
        long long nk_slot_shift_;                                           \
        if (!::nk::batch_slot((G), nk_slot_shift_)) return;                  \
        if (nk_slot_shift_) ::nk::rebase_all(nk_slot_shift_, __VA_ARGS__);   \
    }

// ---- host side helpers ------------------------------------------------------------------------------------
// Slots of the batched launch being captured on this host thread (1 outside); the grid helpers below give every
// launch that many z blocks.
int batch_slots();
void set_batch_slots(int n);
// Sets the slot count for the lifetime of the scope (graph capture of a batch).
struct BatchScope {
    explicit BatchScope(int n) { set_batch_slots(n); }
    ~BatchScope() { set_batch_slots(1); }
    BatchScope(const BatchScope&) = delete;
    BatchScope& operator=(const BatchScope&) = delete;
};
// Kernels launched by the library in this process (instrumentation; every launch site calls count_launch()).
void count_launch();
void count_launches(long long n);
void set_capturing(bool on);
long long launch_count();

// ---- host side helpers (continued) ------------------------------------------------------------------------------
struct LaunchDims {
    dim3 grid, block;
};
constexpr int SM_COUNT = 152;
// Shape of the conjugate-gradient vector kernels: a warp takes the row segments (32 columns of one row) t, t + warps of the
// grid, ... and a block adds its sums once.  The FP64 pipe is one per SM: a small grid spreads one or two warps over every
// SM, a large one has as many warps resident as hide its loads, each SM with the same work to its end.  k_cg_update:
// 128 x 64 10.3 -> 7.6 us, 1024 x 512 22.6 us without and 18.4 us with the r.z_old of the flexible beta.
inline LaunchDims vec_dims(int nx, int ny) {
    const long long w = (long long)((nx + 31) / 32) * ny;
    const int warps = w <= 2ll * SM_COUNT ? 1 : (w <= 4ll * SM_COUNT ? 2 : (w <= 8ll * SM_COUNT ? 4 : 8));
    const long long blocks = (w + warps - 1) / warps, resident = 3ll * SM_COUNT;
    LaunchDims d;
    d.block = dim3(32, warps);
    d.grid = dim3((unsigned)(blocks < resident ? blocks : resident), 1, batch_slots());
    return d;
}
// Calls body(k, ok) for the thread's cells, two row segments at a time: their indices k[2] and whether they exist, ok[2].
template <typename F>
__device__ __forceinline__ void for_each_cell_pair(int Nx, int Ny, int pitch, F&& body) {
    const int across = (Nx + 31) / 32, n = across * Ny, step = (int)(gridDim.x * blockDim.y);
    for (int t = (int)(threadIdx.y * gridDim.x + blockIdx.x); t < n; t += 2 * step) {
        int k[2];
        bool ok[2];
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const int s = t + a * step, j = s / across, i = (s - j * across) * 32 + (int)threadIdx.x;
            ok[a] = s < n && i < Nx;
            k[a] = j * pitch + i;
        }
        body(k, ok);
    }
}
inline LaunchDims dims2d(int nx, int ny) {
    LaunchDims d;
    d.block = dim3(BX, BY);
    d.grid = dim3((nx + BX - 1) / BX, (ny + BY - 1) / BY, batch_slots());
    return d;
}

}  // namespace nk
