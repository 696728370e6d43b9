// nk_cluster.cu — the coarse levels of the multigrid V-cycle in one thread-block cluster.
//
// A level of a few thousand cells is a microsecond of arithmetic on a few SMs, but a grid-wide launch per sweep costs
// 3.5-9 us of launch, index and load latency whatever its size.  From the first level that fits down to the coarsest,
// the whole rest of v_cycle! (multigrid_preconditioner.jl:144-163) runs here: pre-sweeps from zero, residual,
// restriction, the coarsest sweeps, prolongation, post-sweeps.
//
// Layout.  The CTAs of the cluster split the rows of every level.  A thread keeps its cells' iterate and the scaled
// stencil rows in registers, and the masked iterate lives in shared memory with a one-point halo (two buffers per
// level, all levels resident).  A sweep reads seven neighbours from its own CTA's buffer, writes the other buffer, and
// pushes its first and last row into the neighbour CTAs' halo rows through distributed shared memory.  Restriction and
// prolongation read the other level's rows wherever they live.
//
// Arithmetic.  A sweep is x' = x + w (b - A x) with w = 1 / rowsum.  A row of A couples five points of its own component
// and four of the other, and its nine coefficients change only with the coefficients, so -A is formed once per solve
// (k_inverse_row_sum, nk_solver.cu) and a sweep costs twenty multiply-adds and twelve subtractions a cell: as in the
// grid-wide kernels neighbours are differenced before they are multiplied, so that a residual rounds at the size of its own
// terms and not of rowsum |x|.  (Sums of products of whole values cost twelve operations less, 44.2 against 44.7 us a CG step
// of 128 x 64, 67.8 against 68.3 of 320 x 160 DIVA, 150 against 160 of 300 x 180 FP64, and left a smooth mode wrong by 2e-5
// in FP32 where differences leave 1e-6, tests/test_gpu_preconditioner_edges.py.)
// The residual is the sweep's own b - A x: a prescribed row, whose w is zero, keeps its b in it.
//
// What binds it: latency, a sweep being seven shared loads, the multiply-adds and one cluster barrier.  Split: sixteen
// CTAs of 512 threads with one cell a thread where the level allows beat eight CTAs (128 x 64 solve 66.8 against 70.5 us a
// CG iteration, 320 x 160 DIVA 109.9 against 125.9), 256 threads (71.7) and levels of 1024 cells kept inside the first CTA, without cluster barriers but with
// its one shared-memory pipe (72.4).
// Measured, a whole CG iteration, grid-wide launches with the former one-block coarsest kernel against this one:
// 128 x 64 mixed 105 -> 67 us, 320 x 160 DIVA 182 -> 110, 1024 x 512 297 -> 254, 300 x 180 FP64 203 -> 167 (with the other
// kernels of a step as they are now 108, 130, 224 and 189 without it, 43, 70, 153 and 162 with it).  Where the cluster
// holds the finest level too it also takes the step's r.z: 128 x 64 mixed 51 -> 48 us against a pass of its own.
#include <cooperative_groups.h>

#include "nk_kernels.cuh"
#include "nk_transfer.cuh"

namespace nk {

namespace cg = cooperative_groups;

constexpr int CLUSTER_THREADS = 512;
constexpr int CLUSTER_MAX_CTAS = 16;             // the largest cluster (above 8 by an opt-in attribute)
constexpr int CLUSTER_CTA_CELLS = 256;           // cells of the top level per CTA, until the cluster is full
constexpr size_t CLUSTER_SMEM_LIMIT = 200 * 1024;

constexpr int CLUSTER_MAX_ROWS = 1000;           // (j magic) >> 20 divides exactly while j * rows < 2^20

constexpr int CLUSTER_MAX_HALO = 8;

// Cells a thread may own.  A cell's stencil, right-hand side and iterate take 26 registers in FP32 and 52 in FP64, of
// the 128 a thread has; four cells in FP32 spilled (1360 bytes) and were slower than leaving the level to the grid.
template <typename T>
constexpr int cluster_max_cells() { return sizeof(T) == 4 ? 2 : 1; }

// Cells a CTA of the coarsest level in FP64.  Its twenty sweeps are the FP64 pipe's, sixteen SMs against all of them: a CG step
// with that level alone takes 92 us in the cluster and 97 grid-wide at 64 x 96 (384 cells a CTA), 99 and 96 at 100 x 64 (400),
// 103 and 97 at 64 x 112 (448), 113 and 95 at 128 x 64 (512); on cells that are not square 94 and 105, 100 and 107, 104 and
// 106, 114 and 105.  A finer level of 512 cells a CTA takes four sweeps and saves its transfers' launches: 256 x 128, with
// 128 x 64 and three more in the cluster, 156 against 258 us.
constexpr int CLUSTER_FP64_COARSEST = 384;

// One level as a CTA of the cluster sees it.
template <typename T>
struct ClusterLevel {
    using V2 = typename Vec2<T>::type;
    using V4 = typename Vec4<T>::type;
    int Nx, Ny, pitch, px, py, cx, cy;
    V2* x; V2* b; const V4* st; const uint8_t* mask;
    int rows, W, off, size;    // rows per CTA, padded row length, offset of the two buffers, entries of one
    unsigned magic;
    int j0, cnt;               // this CTA's first row and number of rows
    int south, north;          // ranks that hold the rows below and above (-1: none, the halo stays zero)
    int south_row;             // row index, in the buffers of `south`, of its north halo
    __device__ __forceinline__ int owner(int j) const { return (int)(((unsigned)j * magic) >> 20); }
    __device__ __forceinline__ int count(int rank) const { int c = Ny - rank * rows; return c < 0 ? 0 : (c > rows ? rows : c); }
};

template <typename T>
__device__ __forceinline__ ClusterLevel<T> cluster_level(const ClusterLevels<T>& C, int l, int rank, long long d) {
    ClusterLevel<T> K;
    const LevelView<T>& L = C.lv[l];
    K.Nx = L.o.g.Nx; K.Ny = L.o.g.Ny; K.pitch = L.o.g.pitch; K.px = L.o.g.px; K.py = L.o.g.py;
    K.cx = L.cx; K.cy = L.cy;
    K.x = L.x; K.b = L.b; K.st = L.st; K.mask = L.o.mask;
    rebase_all(d, K.x, K.b, K.st, K.mask);
    K.rows = C.rows[l];
    K.magic = C.magic[l];
    K.off = C.off[l];
    K.W = K.Nx + 2;
    K.size = (K.rows + 2) * K.W;
    K.j0 = rank * K.rows;
    K.cnt = K.count(rank);
    K.south = K.north = -1;
    K.south_row = 0;
    if (K.cnt > 0) {
        int js = K.j0 - 1, jn = K.j0 + K.cnt;
        if (js < 0 && K.py) js = K.Ny - 1;
        if (jn >= K.Ny) jn = K.py ? 0 : -1;
        if (js >= 0) { K.south = K.owner(js); K.south_row = K.count(K.south) + 1; }
        if (jn >= 0) K.north = K.owner(jn);
    }
    return K;
}

// A thread's cells of one level: the iterate, b, w and the rows of -A (stencil_rows, nk_solver.cu), so that a sweep is a
// chain of multiply-adds over differences of neighbours.
template <typename T, int CPT>
struct ClusterCells {
    using V2 = typename Vec2<T>::type;
    V2 x[CPT], b[CPT], w[CPT];
    T u[CPT][9], v[CPT][9];
    int p[CPT];                // index in a buffer, -1 for no cell
    unsigned flags[CPT];
};
constexpr unsigned CELL_U = 1, CELL_V = 2;            // the component takes part in the strain rates
constexpr unsigned CELL_WEST = 4, CELL_EAST = 8;      // first / last column of a periodic axis: repeated in the pad
constexpr unsigned CELL_SOUTH = 16, CELL_NORTH = 32;  // first / last row of the CTA: pushed into the neighbour's halo
constexpr unsigned CELL_IU = 64, CELL_IV = 128;       // identity rows
constexpr int CELL_COL = 8;                           // the column index starts at this bit

template <typename T, int CPT>
__device__ __forceinline__ int cell_i(const ClusterCells<T, CPT>& c, int k) { return (int)(c.flags[k] >> CELL_COL); }

// The cells' places, stencil rows and weights w = 1 / rowsum.
template <typename T, int CPT>
__device__ __forceinline__ void cluster_setup(const ClusterLevel<T>& K, ClusterCells<T, CPT>& c) {
    using V4 = typename Vec4<T>::type;
    const int n = K.cnt * K.Nx, plane = K.Nx * K.Ny;
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
        const int e = (int)threadIdx.x + k * CLUSTER_THREADS;
        c.p[k] = -1;
        c.flags[k] = 0;
        if (e >= n) continue;
        const int jl = e / K.Nx, i = e - jl * K.Nx;
        c.p[k] = (jl + 1) * K.W + i + 1;
        const uint8_t m = __ldg(K.mask + (K.j0 + jl) * K.pitch + i);
        const V4* st = K.st + K.j0 * K.Nx + e;
        V4 a = st[0], b = st[plane], f = st[2 * plane], h = st[3 * plane], o = st[4 * plane];
        T* u = c.u[k];
        T* v = c.v[k];
        u[0] = a.x; u[1] = a.y; u[2] = a.z; u[3] = a.w; u[4] = b.x; u[5] = b.y; u[6] = b.z; u[7] = b.w; u[8] = o.x;
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w; v[4] = h.x; v[5] = h.y; v[6] = h.z; v[7] = h.w; v[8] = o.y;
        c.w[k].x = o.z;
        c.w[k].y = o.w;
        c.flags[k] = ((m & U_INACTIVE) ? 0u : CELL_U) | ((m & V_INACTIVE) ? 0u : CELL_V) | ((K.px && i == 0) ? CELL_WEST : 0u) |
                     ((K.px && i == K.Nx - 1) ? CELL_EAST : 0u) | ((jl == 0 && K.south >= 0) ? CELL_SOUTH : 0u) |
                     ((jl == K.cnt - 1 && K.north >= 0) ? CELL_NORTH : 0u) | ((m & U_IDENTITY) ? CELL_IU : 0u) |
                     ((m & V_IDENTITY) ? CELL_IV : 0u) | ((unsigned)i << CELL_COL);
    }
}
// b - A x of cell k from the masked iterate in `in`
template <typename T, int CPT>
__device__ __forceinline__ typename Vec2<T>::type cluster_residual(const ClusterLevel<T>& K, const ClusterCells<T, CPT>& c, int k,
                                                                   const typename Vec2<T>::type* in) {
    using V2 = typename Vec2<T>::type;
    const V2* q = in + c.p[k];
    V2 E = q[1], Wt = q[-1], N = q[K.W], S = q[-K.W], NW = q[K.W - 1], SE = q[1 - K.W];
    T mu = (c.flags[k] & CELL_U) ? c.x[k].x : T(0), mv = (c.flags[k] & CELL_V) ? c.x[k].y : T(0);
    const T* u = c.u[k];
    const T* v = c.v[k];
    const T nc = N.y - mv, wc = Wt.y - mv, ec = E.x - mu, sc = S.x - mu;   // in both rows
    V2 r;
    if constexpr (sizeof(T) == 8) {   // the FP64 pipe: one chain, with no additions of its own (300 x 180: 162 us a CG step, 169 with three)
        r.x = c.b[k].x + u[4] * c.x[k].x + u[0] * ec + u[1] * (Wt.x - mu) + u[2] * (N.x - mu) + u[3] * sc + u[5] * nc +
              u[6] * (Wt.y - NW.y) + u[7] * (N.y - NW.y) + u[8] * wc;
        r.y = c.b[k].y + v[4] * c.x[k].y + v[0] * nc + v[1] * (S.y - mv) + v[2] * (E.y - mv) + v[3] * wc + v[5] * ec +
              v[6] * (S.x - SE.x) + v[7] * (E.x - SE.x) + v[8] * sc;
    } else {                          // FP32, latency: three short ones
        T ya = c.b[k].x + u[4] * c.x[k].x + u[0] * ec + u[1] * (Wt.x - mu), yb = u[5] * nc + u[6] * (Wt.y - NW.y) + u[7] * (N.y - NW.y) + u[8] * wc;
        T za = c.b[k].y + v[4] * c.x[k].y + v[0] * nc + v[1] * (S.y - mv), zb = v[5] * ec + v[6] * (S.x - SE.x) + v[7] * (E.x - SE.x) + v[8] * sc;
        r.x = ya + (yb + (u[2] * (N.x - mu) + u[3] * sc));
        r.y = za + (zb + (v[2] * (E.y - mv) + v[3] * wc));
    }
    return r;
}
// The first sweep of cell k, from zero, and a further one from the masked iterate in `in`
template <typename T, int CPT>
__device__ __forceinline__ void cluster_first(ClusterCells<T, CPT>& c, int k) {
    c.x[k].x = c.w[k].x * c.b[k].x;
    c.x[k].y = c.w[k].y * c.b[k].y;
}
template <typename T, int CPT>
__device__ __forceinline__ void cluster_sweep(const ClusterLevel<T>& K, ClusterCells<T, CPT>& c, int k, const typename Vec2<T>::type* in) {
    const auto r = cluster_residual<T, CPT>(K, c, k, in);
    c.x[k].x += c.w[k].x * r.x;
    c.x[k].y += c.w[k].y * r.y;
}

// Cell k's masked pair m into buffer `buf` (offset from the start of shared memory), its periodic copies, and the halo
// rows of the neighbour CTAs.
template <typename T, int CPT>
__device__ __forceinline__ void cluster_put(cg::cluster_group& cl, typename Vec2<T>::type* sm, const ClusterLevel<T>& K, int buf,
                                            const ClusterCells<T, CPT>& c, int k, typename Vec2<T>::type m) {
    using V2 = typename Vec2<T>::type;
    const unsigned f = c.flags[k];
    const int p = c.p[k], Nx = K.Nx;
    V2* b = sm + buf;
    b[p] = m;
    if (f & CELL_WEST) b[p + Nx] = m;
    if (f & CELL_EAST) b[p - Nx] = m;
    if (f & (CELL_SOUTH | CELL_NORTH)) {
        const int col = cell_i<T, CPT>(c, k) + 1;
        if (f & CELL_SOUTH) {   // this row is the north halo of the CTA below
            V2* r = cl.map_shared_rank(b, K.south) + K.south_row * K.W + col;
            *r = m;
            if (f & CELL_WEST) r[Nx] = m;
            if (f & CELL_EAST) r[-Nx] = m;
        }
        if (f & CELL_NORTH) {   // and the south halo of the CTA above
            V2* r = cl.map_shared_rank(b, K.north) + col;
            *r = m;
            if (f & CELL_WEST) r[Nx] = m;
            if (f & CELL_EAST) r[-Nx] = m;
        }
    }
}
template <typename T, int CPT>
__device__ __forceinline__ typename Vec2<T>::type cluster_masked(const ClusterCells<T, CPT>& c, int k, typename Vec2<T>::type x) {
    if (!(c.flags[k] & CELL_U)) x.x = T(0);
    if (!(c.flags[k] & CELL_V)) x.y = T(0);
    return x;
}

// Row j of level K's buffer, in whichever CTA holds it: column i is entry i + 1
template <typename T>
__device__ __forceinline__ const typename Vec2<T>::type* cluster_row(cg::cluster_group& cl, typename Vec2<T>::type* sm,
                                                                    const ClusterLevel<T>& K, int buf, int j) {
    const int rank = K.owner(j);
    return cl.map_shared_rank(sm + buf, rank) + (j - rank * K.rows + 1) * K.W + 1;
}

// The fine points 2 I - 1 .. 2 I + 2 (I alone on an axis that is not halved) of one axis of the restriction: their
// indices and the weights of a face-located and of a centre-located component (ridx and rweight of nk_transfer.cuh, whose
// rule this writes out for four points at once; a point beyond a Bounded
// edge has weight zero and reads the edge).
template <typename T>
__device__ __forceinline__ void restriction_axis(int I, int Nc, int Nf, bool periodic, int c, int* at, T* face, T* centre) {
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (c == 1) {
            at[a] = I;
            face[a] = centre[a] = a == 1 ? T(1) : T(0);
        } else {
            int i = 2 * I + a - 1;
            at[a] = periodic ? (i < 0 ? i + Nf : (i >= Nf ? i - Nf : i)) : (i < 0 ? 0 : (i > Nf - 1 ? Nf - 1 : i));
            face[a] = a == 1 ? T(1) : (a == 3 || (a == 0 && !periodic && I == 0) ? T(0) : T(1) / T(2));
            T w = a == 1 || a == 2 ? T(3) / T(4) : T(1) / T(4);
            if (!periodic) {
                if ((I == 0 && a == 0) || (I == Nc - 1 && a == 3)) w = T(0);
                if ((I == 0 && a == 1) || (I == Nc - 1 && a == 2)) w += T(1) / T(4);
            }
            centre[a] = w;
        }
    }
}

// The sweeps of the coarsest level with `halo` rows of the neighbours swept along, one cell a thread: the rows that are right
// shrink by one a sweep on either side, and only when a CTA's own are next does it take the halo anew, for one cluster
// barrier in `halo` sweeps instead of one a sweep (894 cycles a sweep, 700 of them the barrier): a CG step of 128 x 64 mixed
// 47.2 -> 43.8 us, of 320 x 160 DIVA 72.6 -> 70.7, of 1024 x 512 156.5 -> 153.5.  As many rows as one cell a thread allows, up
// to 8 (the next would save a barrier in 72 sweeps).  `c` are the CTA's own cells
// with b in place; their iterate goes to c.x and, masked, to the level's first buffer.  FP32 only: the rows that
// several CTAs sweep would be paid for on the FP64 pipe.
template <typename T, int CPT>
__device__ __forceinline__ void coarsest_window(cg::cluster_group& cl, typename Vec2<T>::type* sm, const ClusterLevels<T>& C,
                                                const ClusterLevel<T>& K, ClusterCells<T, CPT>& c, int rank) {
    using V2 = typename Vec2<T>::type;
    using V4 = typename Vec4<T>::type;
    const int Nx = K.Nx, halo = C.halo, own = K.cnt * Nx, share = K.rows * Nx, size = (K.rows + 2 * halo + 2) * K.W;
    V2* const shared_rows = sm + C.window;            // the own rows as the neighbours read them, twice
    V2* const x0 = shared_rows + 2 * share;
    const int tid = threadIdx.x;
    if (tid < own) shared_rows[tid] = c.b[0];         // (share >= own: one cell a thread)
    int lo = K.j0 - halo, hi = K.j0 + K.cnt + halo;
    if (!K.py) { lo = lo < 0 ? 0 : lo; hi = hi > K.Ny ? K.Ny : hi; }
    if (K.cnt == 0) hi = lo;
    const int row = tid / Nx, i = tid - row * Nx, jw = lo + row;
    const bool in = jw < hi;
    int j = jw % K.Ny;
    if (j < 0) j += K.Ny;
    const int far = jw < K.j0 ? K.j0 - jw : (jw >= K.j0 + K.cnt ? jw - (K.j0 + K.cnt - 1) : 0);   // rows from the own ones
    ClusterCells<T, 1> z;
    z.p[0] = (row + 1) * K.W + i + 1;
    z.flags[0] = 0;
    int from = 0;
    if (in) {
        const uint8_t m = __ldg(K.mask + j * K.pitch + i);
        const int plane = Nx * K.Ny;
        const V4* st = K.st + j * Nx + i;
        const V4 a = st[0], b = st[plane], f = st[2 * plane], h = st[3 * plane], o = st[4 * plane];
        T *u = z.u[0], *v = z.v[0];
        u[0] = a.x; u[1] = a.y; u[2] = a.z; u[3] = a.w; u[4] = b.x; u[5] = b.y; u[6] = b.z; u[7] = b.w; u[8] = o.x;
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w; v[4] = h.x; v[5] = h.y; v[6] = h.z; v[7] = h.w; v[8] = o.y;
        z.w[0].x = o.z;
        z.w[0].y = o.w;
        z.flags[0] = ((m & U_INACTIVE) ? 0u : CELL_U) | ((m & V_INACTIVE) ? 0u : CELL_V);
        from = K.owner(j);
    }
    const int at = (j - from * K.rows) * Nx + i;      // the cell in its CTA's shared_rows
    auto put = [&](int buf) {
        V2 *b = x0 + buf * size + z.p[0], m = cluster_masked<T, 1>(z, 0, z.x[0]);
        b[0] = m;
        if (K.px && i == 0) b[Nx] = m;
        if (K.px && i == Nx - 1) b[-Nx] = m;
    };
    cl.sync();
    if (in) {                                         // the first sweep from zero: x = w b
        z.b[0] = cl.map_shared_rank(shared_rows, from)[at];
        cluster_first<T, 1>(z, 0);
        put(0);
    }
    __syncthreads();
    int cur = 0, depth = halo, turn = 1;
    for (int s = 1; s < C.coarsest; ++s) {
        if (depth == 0) {
            V2* const rows = shared_rows + turn * share;   // the other one may still be read
            if (in && far == 0) rows[at] = z.x[0];
            cl.sync();
            if (in && far > 0) {
                z.x[0] = cl.map_shared_rank(rows, from)[at];
                put(cur);
            }
            __syncthreads();
            turn ^= 1;
            depth = halo;
        }
        --depth;
        if (in && far <= depth) {
            cluster_sweep<T, 1>(K, z, 0, x0 + cur * size);
            put(cur ^ 1);
        }
        __syncthreads();
        cur ^= 1;
    }
    V2* const result = shared_rows + turn * share;    // the one that no CTA reads any more
    if (in && far == 0) {
        result[at] = z.x[0];
        const V2 m = cluster_masked<T, 1>(z, 0, z.x[0]);
        V2* b = sm + K.off + (jw - K.j0 + 1) * K.W + i + 1;
        b[0] = m;
        if (K.px && i == 0) b[Nx] = m;
        if (K.px && i == Nx - 1) b[-Nx] = m;
    }
    cl.sync();
    if (tid < own) c.x[0] = result[tid];
}

template <typename T, int CPT>
__global__ void __launch_bounds__(CLUSTER_THREADS, 1) k_coarse_cluster(const __grid_constant__ ClusterLevels<T> C, const int* done, CGDot dot) {
    long long d;
    if (!batch_slot(C.lv[0].o.g, d)) return;   // the same answer in every CTA of a cluster (one slot)
    if (d) { rebase(done, d); rebase(dot, d); }
    if (done && *(volatile const int*)done) return;
    using V2 = typename Vec2<T>::type;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = blockIdx.x, last = C.n - 1;
    extern __shared__ __align__(32) unsigned char smem_raw[];
    V2* sm = reinterpret_cast<V2*>(smem_raw);

    ClusterCells<T, CPT> c;
    ClusterLevel<T> K = cluster_level(C, 0, rank, d);
    cluster_setup<T, CPT>(K, c);
#pragma unroll
    for (int k = 0; k < CPT; ++k)
        if (c.p[k] >= 0) {
            const int e = (int)threadIdx.x + k * CLUSTER_THREADS, i = cell_i<T, CPT>(c, k);
            c.b[k] = K.b[(K.j0 + (e - i) / K.Nx) * K.pitch + i];
        }
    for (int e = threadIdx.x; e < C.total; e += CLUSTER_THREADS) { V2 z; z.x = z.y = T(0); sm[e] = z; }
    cl.sync();   // the zeroed halos are in place before a neighbour writes into them
    // down
    for (int l = 0;; ++l) {
        const int buf0 = K.off, buf1 = K.off + K.size;
        const int ns = l == last ? C.coarsest : C.sweeps;
        if constexpr (sizeof(T) == 4)
            if (l == last && C.halo) {
                coarsest_window<T, CPT>(cl, sm, C, K, c, rank);
                break;
            }
#pragma unroll
        for (int k = 0; k < CPT; ++k)   // the first sweep from zero: x = w b
            if (c.p[k] >= 0) {
                cluster_first<T, CPT>(c, k);
                cluster_put<T, CPT>(cl, sm, K, buf0, c, k, cluster_masked<T, CPT>(c, k, c.x[k]));
            }
        cl.sync();
        int cur = buf0;
        for (int s = 1; s < ns; ++s) {
            const int nxt = cur == buf0 ? buf1 : buf0;
#pragma unroll
            for (int k = 0; k < CPT; ++k)
                if (c.p[k] >= 0) {
                    cluster_sweep<T, CPT>(K, c, k, sm + cur);
                    cluster_put<T, CPT>(cl, sm, K, nxt, c, k, cluster_masked<T, CPT>(c, k, c.x[k]));
                }
            cl.sync();
            cur = nxt;
        }
        if (l == last) break;
        const int res = cur == buf0 ? buf1 : buf0;   // the residual takes the free buffer
#pragma unroll
        for (int k = 0; k < CPT; ++k)
            if (c.p[k] >= 0) sm[res + c.p[k]] = cluster_masked<T, CPT>(c, k, cluster_residual<T, CPT>(K, c, k, sm + cur));
        ClusterLevel<T> N = cluster_level(C, l + 1, rank, d);
        cluster_setup<T, CPT>(N, c);
        cl.sync();
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            if (c.p[k] < 0) continue;
            const int e = (int)threadIdx.x + k * CLUSTER_THREADS, I = cell_i<T, CPT>(c, k), J = N.j0 + (e - I) / N.Nx;
            int at[4], row[4];
            T fx[4], cx[4], fy[4], cy[4];
            restriction_axis<T>(I, N.Nx, K.Nx, K.px, N.cx, at, fx, cx);
            restriction_axis<T>(J, N.Ny, K.Ny, K.py, N.cy, row, fy, cy);
            T su = T(0), sv = T(0);
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const V2* r = cluster_row<T>(cl, sm, K, res, row[b]);
                T hu = T(0), hv = T(0);
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    V2 q = r[at[a]];
                    if (a < 3) hu += fx[a] * q.x;
                    hv += cx[a] * q.y;
                }
                su += cy[b] * hu;
                if (b < 3) sv += fy[b] * hv;
            }
            V2 b;
            b.x = (c.flags[k] & CELL_IU) ? T(0) : su;
            b.y = (c.flags[k] & CELL_IV) ? T(0) : sv;
            N.b[J * N.pitch + I] = b;   // read back by this thread on the way up
            c.b[k] = b;
        }
        K = N;
    }
    // up: the coarser level's iterate is in the buffer its last sweep wrote
    int coarse_buf = K.off + (!C.halo && ((C.coarsest - 1) & 1) ? K.size : 0);
    for (int l = last - 1; l >= 0; --l) {
        ClusterLevel<T> N = cluster_level(C, l, rank, d);
        cluster_setup<T, CPT>(N, c);
        const int down = (C.sweeps - 1) & 1;   // the buffer that holds the iterate of the way down
        int cur = N.off + (down ? 0 : N.size);
        const int old = N.off + (down ? N.size : 0);
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            if (c.p[k] < 0) continue;
            const int e = (int)threadIdx.x + k * CLUSTER_THREADS, i = cell_i<T, CPT>(c, k), j = N.j0 + (e - i) / N.Nx;
            V2 x = sm[old + c.p[k]];
            c.b[k] = N.b[j * N.pitch + i];
            // an inactive row is an identity row: its iterate is w b after every sweep, and shared memory holds zero
            if (!(c.flags[k] & CELL_U)) x.x = c.w[k].x * c.b[k].x;
            if (!(c.flags[k] & CELL_V)) x.y = c.w[k].y * c.b[k].y;
            int fi1, fi2, ci1, ci2, fj1, fj2, cj1, cj2;   // face and centre parents of each axis
            T fa1, fa2, ca1, ca2, fb1, fb2, cb1, cb2;
            parents<T>(i, K.Nx, K.px, true, K.cx, fi1, fi2, fa1, fa2);
            parents<T>(i, K.Nx, K.px, false, K.cx, ci1, ci2, ca1, ca2);
            parents<T>(j, K.Ny, K.py, true, K.cy, fj1, fj2, fb1, fb2);
            parents<T>(j, K.Ny, K.py, false, K.cy, cj1, cj2, cb1, cb2);
            if (fj2 >= K.Ny) { fj2 = fj1; fb2 = T(0); }   // the north wall face of a Bounded axis carries zero
            const V2 *ru1 = cluster_row<T>(cl, sm, K, coarse_buf, cj1), *ru2 = cluster_row<T>(cl, sm, K, coarse_buf, cj2);
            const V2 *rv1 = cluster_row<T>(cl, sm, K, coarse_buf, fj1), *rv2 = cluster_row<T>(cl, sm, K, coarse_buf, fj2);
            T pu = fa1 * (cb1 * ru1[fi1].x + cb2 * ru2[fi1].x) + fa2 * (cb1 * ru1[fi2].x + cb2 * ru2[fi2].x);
            T pv = ca1 * (fb1 * rv1[ci1].y + fb2 * rv2[ci1].y) + ca2 * (fb1 * rv1[ci2].y + fb2 * rv2[ci2].y);
            if (!(c.flags[k] & CELL_IU)) x.x += pu;
            if (!(c.flags[k] & CELL_IV)) x.y += pv;
            c.x[k] = x;
            cluster_put<T, CPT>(cl, sm, N, cur, c, k, cluster_masked<T, CPT>(c, k, x));
        }
        cl.sync();
        for (int s = 0; s < C.sweeps; ++s) {
            const int nxt = cur == N.off ? N.off + N.size : N.off;
            const bool out = l == 0 && s == C.sweeps - 1;
#pragma unroll
            for (int k = 0; k < CPT; ++k)
                if (c.p[k] >= 0) {
                    cluster_sweep<T, CPT>(N, c, k, sm + cur);
                    if (!out) cluster_put<T, CPT>(cl, sm, N, nxt, c, k, cluster_masked<T, CPT>(c, k, c.x[k]));
                }
            if (!out) cl.sync();
            cur = nxt;
        }
        coarse_buf = cur;
        K = N;
    }
    double rz = 0.0;
    const int ze = dot.r && sizeof(T) == 4 ? dot.sc->r32_exp : 0;
#pragma unroll
    for (int k = 0; k < CPT; ++k)
        if (c.p[k] >= 0) {
            const int e = (int)threadIdx.x + k * CLUSTER_THREADS, i = cell_i<T, CPT>(c, k);
            const int q = (K.j0 + (e - i) / K.Nx) * K.pitch + i;
            K.x[q] = c.x[k];
            if (dot.r) {   // z = x 2^ze
                const double2 r = dot.r[q];
                if constexpr (sizeof(T) == 4) rz = fma(r.x, widen_pow2(c.x[k].x, ze), fma(r.y, widen_pow2(c.x[k].y, ze), rz));
                else rz = fma(r.x, c.x[k].x, fma(r.y, c.x[k].y, rz));
            }
        }
    if (!dot.r) {
        cl.sync();   // no CTA leaves while another may still read its shared memory
        return;
    }
    // the CTA's sum by one warp, then the CTAs' sums in the first CTA: fixed trees
    __shared__ double sums[CLUSTER_THREADS], ctas[CLUSTER_MAX_CTAS];
    sums[threadIdx.x] = rz;
    __syncthreads();
    if (threadIdx.x < 32) {
        double a[CLUSTER_THREADS / 32];
#pragma unroll
        for (int k = 0; k < CLUSTER_THREADS / 32; ++k) a[k] = sums[threadIdx.x + 32 * k];
#pragma unroll
        for (int h = CLUSTER_THREADS / 64; h > 0; h >>= 1)
#pragma unroll
            for (int k = 0; k < h; ++k) a[k] += a[k + h];
        const double t = warp_sum(a[0]);
        if (threadIdx.x == 0) *cl.map_shared_rank(&ctas[rank], 0) = t;
    }
    const CGDotScalars scalars(dot.sc);
    cl.sync();   // the sums are there, and no CTA leaves while another may still read its shared memory
    if (rank == 0 && threadIdx.x < 32) {
        const double t = warp_sum((int)threadIdx.x < C.ctas ? ctas[threadIdx.x] : 0.0);
        if (threadIdx.x == 0) scalars.finish(dot, t);
    }
}

// Rows per CTA and buffer offsets of levels lv[0 .. n-1] (lv[0] the finest of them); false if they do not fit.
template <typename T>
bool cluster_plan(ClusterLevels<T>& C) {
    if (C.n < 1 || C.n > MAX_COARSE_LEVELS || C.sweeps < 1 || C.coarsest < 1) return false;
    long long top = (long long)C.lv[0].o.g.Nx * C.lv[0].o.g.Ny;
    const int ctas = (int)((top + CLUSTER_CTA_CELLS - 1) / CLUSTER_CTA_CELLS);
    C.ctas = 1;
    while (C.ctas < ctas && C.ctas < CLUSTER_MAX_CTAS) C.ctas *= 2;
    long long off = 0;
    C.cells = 1;
    for (int l = 0; l < C.n; ++l) {
        const DevGrid<T>& g = C.lv[l].o.g;
        int rows = (g.Ny + C.ctas - 1) / C.ctas;
        long long cells = (long long)rows * g.Nx;
        if (!C.lv[l].st || g.Ny > CLUSTER_MAX_ROWS || cells > (long long)cluster_max_cells<T>() * CLUSTER_THREADS) return false;
        if (sizeof(T) == 8 && l == C.n - 1 && cells > CLUSTER_FP64_COARSEST) return false;
        int need = (int)((cells + CLUSTER_THREADS - 1) / CLUSTER_THREADS);
        while (C.cells < need) C.cells *= 2;
        C.rows[l] = rows;
        C.magic[l] = ((1u << 20) + rows - 1) / rows;   // j / rows = (j magic) >> 20 for every row j < CLUSTER_MAX_ROWS
        C.off[l] = (int)off;
        off += 2ll * (rows + 2) * (g.Nx + 2);
        if (off * (long long)sizeof(typename Vec2<T>::type) > (long long)CLUSTER_SMEM_LIMIT) return false;
    }
    C.halo = 0;
    if constexpr (sizeof(T) == 4) {
        const DevGrid<T>& g = C.lv[C.n - 1].o.g;
        const int rows = C.rows[C.n - 1], fit = (CLUSTER_THREADS / g.Nx - rows) / 2, halo = fit < CLUSTER_MAX_HALO ? fit : CLUSTER_MAX_HALO;
        const long long window = off + 2ll * rows * g.Nx + 2ll * (rows + 2 * halo + 2) * (g.Nx + 2);
        if (C.ctas > 1 && halo >= 2 && C.coarsest >= 4 && window * (long long)sizeof(typename Vec2<T>::type) <= (long long)CLUSTER_SMEM_LIMIT) {
            C.halo = halo;
            C.window = (int)off;
            off = window;
        }
    }
    C.total = (int)off;
    return true;
}

template <typename T, int CPT>
static void launch_cluster(const ClusterLevels<T>& C, const int* done, const CGDot& dot, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C.ctas, 1, batch_slots());
    cfg.blockDim = dim3(CLUSTER_THREADS);
    cfg.dynamicSmemBytes = (size_t)C.total * sizeof(typename Vec2<T>::type);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C.ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_coarse_cluster<T, CPT>, C, done, dot);
}
template <typename T>
void launch_coarse_cluster(const ClusterLevels<T>& C, const int* done, const CGDot* with, cudaStream_t s) {
    const CGDot dot = with ? *with : CGDot{};
    if constexpr (cluster_max_cells<T>() >= 2) {
        if (C.cells == 2) launch_cluster<T, 2>(C, done, dot, s);
        else launch_cluster<T, 1>(C, done, dot, s);
    } else {
        launch_cluster<T, 1>(C, done, dot, s);
    }
    count_launch();
}
template <typename T, int CPT>
static bool cluster_fits() {
    return cluster_can_be_placed(k_coarse_cluster<T, CPT>, CLUSTER_MAX_CTAS, CLUSTER_THREADS, CLUSTER_SMEM_LIMIT);
}
// The kernels' shared-memory limit and cluster size on the current device (never in a capture), and whether it has room for
// the largest cluster that cluster_plan asks for.
bool coarse_cluster_available() { return cluster_fits<float, 1>() && cluster_fits<float, 2>() && cluster_fits<double, 1>(); }

template bool cluster_plan<float>(ClusterLevels<float>&);
template bool cluster_plan<double>(ClusterLevels<double>&);
template void launch_coarse_cluster<float>(const ClusterLevels<float>&, const int*, const CGDot*, cudaStream_t);
template void launch_coarse_cluster<double>(const ClusterLevels<double>&, const int*, const CGDot*, cudaStream_t);

}  // namespace nk
