// nk_vcycle.cu — the two halves of a multigrid level in one pass each, for the FP32 hierarchy.
//
// v_cycle! (multigrid_preconditioner.jl:144-163) visits a level with two smoothing sweeps from zero, the residual and its
// restriction on the way down, and with the prolongation and two sweeps on the way up.  As separate launches that reads
// the coefficients, b, 1/rowsum and x five times and costs six launches of 4-10 us a level.  Here a warp walks down the
// grid (Stage, nk_strip.cuh) with the stages of one half one row behind each other in its registers: the row it
// loads enters the first stage, that stage's row above enters the second, and so on; nothing between the stages is
// stored.  Neighbouring columns come by shuffles, so each stage costs a lane on either side (a warp writes 26 columns of the way
// down and 28 of the way up), and a walk starts a few rows above its own.
//
// What binds it: the latency of a warp's instructions (a row is about 150, four cycles apart in one warp), so the reads
// carry no range tests (LevelColumn), run three rows ahead, and the rows in flight are four named slots that need no moves.
// Measured, the six launches against these two: 1024 x 512 50 -> 29 us, 512 x 256 32 -> 16, 256 x 128 28 -> 14; a whole
// 1024 x 512 solve 431 -> 339 ms, 2560 x 320 16.8 -> 13.2.  (With range tests and one row ahead: 45, 23, 20 us.)
#include "nk_kernels.cuh"
#include "nk_transfer.cuh"

namespace nk {

constexpr int DOWN_COLS = 26, DOWN_FIRST = 3;   // columns written by a warp: lanes 3 .. 28, the first even
constexpr int UP_COLS = 28, UP_FIRST = 2;       // lanes 2 .. 29
constexpr int VCYCLE_WARPS = 4;                 // warps per block, side by side

// A lane's column of a level.  Rows and columns beyond a Bounded edge are read at the nearest stored point (0 .. N, whose
// last row and column are the walls) and flagged inactive below 0, where the stored mask does not say so: their velocities
// then read as zero, and no row that is written depends on the coefficients there.
template <typename T>
struct LevelColumn {
    using V2 = typename Vec2<T>::type;
    using V4 = typename Vec4<T>::type;
    struct Row { V2 b, w, x; V4 c; unsigned m; };
    const LevelView<T>& L;
    int i, iw;
    unsigned low;        // both components inactive: the lane's column is below a Bounded edge
    T wall_x, au, av;    // shear factor of the lane's corners; face areas of a regular square grid
    __device__ __forceinline__ LevelColumn(const LevelView<T>& level, int col) : L(level), i(col) {
        const DevGrid<T>& g = L.o.g;
        iw = g.px ? wrapn(i, g.Nx) : (i < 0 ? 0 : (i > g.Nx ? g.Nx : i));
        low = !g.px && i < 0 ? U_INACTIVE | V_INACTIVE : 0u;
        wall_x = !g.px && (i <= 0 || i >= g.Nx) ? L.o.wall_factor : T(1);
        au = av = g.h * g.h;
    }
    __device__ __forceinline__ int row(int j) const {   // the stored row of j (vcycle_rows_wrap_once)
        const DevGrid<T>& g = L.o.g;
        if (g.py) return j < 0 ? j + g.Ny : (j >= g.Ny ? j - g.Ny : j);
        return j < 0 ? 0 : (j > g.Ny ? g.Ny : j);
    }
    __device__ __forceinline__ int face(int j) const { return !L.o.g.py && j < 0 ? 0 : row(j) + 1; }   // Stage::push's jf
    template <bool WITH_X>
    __device__ __forceinline__ void fetch(Row& r, int j, const V2* __restrict__ x) const {
        const DevGrid<T>& g = L.o.g;
        const int k = row(j) * g.pitch + iw;
        r.c = L.o.coef[k];
        r.b = L.b[k];
        r.w = L.irs[k];
        if (WITH_X) r.x = x[k];
        r.m = __ldg(L.o.mask + k);
    }
    // After the row's reads have arrived: (Az β) in place of β, the wall factor in η̄Hᶠᶠ, the inactive flags, and x = w b
    // where the walk starts from zero.  The weight of an inactive row is dropped: its iterate is b already.
    template <bool UNI, bool WITH_X>
    __device__ __forceinline__ void settle(Row& r, int j) const {
        const DevGrid<T>& g = L.o.g;
        if (!UNI) {
            const int jm = row(j);
            const bool in = jm < g.Ny && iw < g.Nx;
            r.c.z *= in ? g.dxf[iw] * g.dyc[jm] : T(0);
            r.c.w *= in ? g.dxc[iw] * g.dyf[jm] : T(0);
        } else {
            r.c.z *= au;
            r.c.w *= av;
        }
        r.c.y *= !g.py && (j <= 0 || j >= g.Ny) ? L.o.wall_factor : wall_x;
        r.m |= low | (!g.py && j < 0 ? U_INACTIVE | V_INACTIVE : 0u);
        if (!WITH_X) {
            r.x.x = r.b.x * r.w.x;
            r.x.y = r.b.y * r.w.y;
        }
        if (r.m & U_INACTIVE) r.w.x = T(0);
        if (r.m & V_INACTIVE) r.w.y = T(0);
    }
};
template <typename T, typename Row>
__device__ __forceinline__ T active_u(const Row& r, T u) { return (r.m & U_INACTIVE) ? T(0) : u; }
template <typename T, typename Row>
__device__ __forceinline__ T active_v(const Row& r, T v) { return (r.m & V_INACTIVE) ? T(0) : v; }

// Two sweeps from zero, the residual and its restriction (full weighting, restrict_at): x2 = both sweeps, C.b = R (b - A x2).
// Only for levels halved in both directions.
template <typename T, bool UNI>
__global__ void __launch_bounds__(32 * VCYCLE_WARPS) k_vcycle_down(LevelView<T> L, LevelView<T> C, typename Vec2<T>::type* __restrict__ x2,
                                                                  int rows, const int* done) {
    NK_BATCH_ENTER(L.o.g, L, C, x2, done)
    if (done && *(volatile const int*)done) return;
    using V2 = typename Vec2<T>::type;
    using Row = typename LevelColumn<T>::Row;
    const DevGrid<T>&g = L.o.g, &cg = C.o.g;
    const int lane = threadIdx.x;
    const int strip = blockIdx.x * VCYCLE_WARPS + threadIdx.y;
    const int J0 = blockIdx.y * rows, J1 = J0 + rows < cg.Ny ? J0 + rows : cg.Ny;
    if (strip * DOWN_COLS >= g.Nx) return;   // whole warp
    const int i = strip * DOWN_COLS - DOWN_FIRST + lane;
    const LevelColumn<T> col(L, i);
    const bool own = lane >= DOWN_FIRST && lane < DOWN_FIRST + DOWN_COLS && i < g.Nx;
    const int I = i >> 1;
    // horizontal weights of the centre-located component at this coarse column (the edges fold, rweight)
    const T w0 = !g.px && I == 0 ? T(1) : T(3) / T(4), w1 = !g.px && I == cg.Nx - 1 ? T(1) : T(3) / T(4);
    V2* const xw = own ? x2 + i : nullptr;
    const bool coarse = own && (i & 1) == 0;
    Stage<T, UNI> s1(g, col.iw), s2(g, col.iw);
    const int ja = 2 * J0 - 3, jb = 2 * J1 + 1;
    Row ring[4];                                    // rows j - 1, j, j + 1 (settled) and j + 2 (in flight)
    V2 x;                                           // x2 of row j - 1, then of row j
    T su = T(0), sv = T(0), nu = T(0), nv = T(0);   // sums of the coarse rows J and J + 1
    col.template fetch<false>(ring[0], ja, nullptr);
    col.template fetch<false>(ring[1], ja + 1, nullptr);
    col.template fetch<false>(ring[2], ja + 2, nullptr);
    col.template settle<UNI, false>(ring[0], ja);
    ring[3] = ring[0];
    s1.mu = active_u<T>(ring[0], ring[0].x.x);
    s1.mv = active_v<T>(ring[0], ring[0].x.y);
    x.x = x.y = T(0);
    auto step = [&](int j, Row& old, Row& cur, Row& nxt) {
        col.template settle<UNI, false>(nxt, j + 1);
        T du, dv;
        s1.push(UNI ? 0 : col.row(j), UNI ? 0 : col.face(j), active_u<T>(nxt, nxt.x.x), active_v<T>(nxt, nxt.x.y), cur.c.x, nxt.c.y, du, dv);
        const V2 prev = x;
        x.x = cur.x.x + (cur.b.x - (cur.c.z * cur.x.x - du)) * cur.w.x;   // the second sweep at row j
        x.y = cur.x.y + (cur.b.y - (cur.c.w * cur.x.y - dv)) * cur.w.y;
        if (xw && j >= 2 * J0 && j < 2 * J1) xw[j * g.pitch] = x;
        const T mx = active_u<T>(cur, x.x), my = active_v<T>(cur, x.y);
        T eu, ev;                                   // the residual of row j - 1
        s2.push(UNI ? 0 : col.row(j - 1), UNI ? 0 : col.face(j - 1), mx, my, old.c.x, cur.c.y, eu, ev);
        const T ru = active_u<T>(old, old.b.x - ((old.m & U_DIRICHLET) ? prev.x : old.c.z * prev.x - eu));
        const T rv = active_v<T>(old, old.b.y - ((old.m & V_DIRICHLET) ? prev.y : old.c.w * prev.y - ev));
        const unsigned full = 0xffffffffu;
        const T rl = __shfl_up_sync(full, ru, 1), rr = __shfl_down_sync(full, ru, 1);
        const T vl = __shfl_up_sync(full, rv, 1), v1 = __shfl_down_sync(full, rv, 1), v2 = __shfl_down_sync(full, rv, 2);
        const T hu = ru + T(1) / T(2) * (rl + rr);
        const T hv = (w0 * rv + w1 * v1) + T(1) / T(4) * (vl + v2);
        const int jr = j - 1, J = jr >> 1;
        if (jr & 1) {            // row 2 J + 1: the last but one of J, the first of J + 1
            su += (!g.py && J == cg.Ny - 1 ? T(1) : T(3) / T(4)) * hu;
            sv += T(1) / T(2) * hv;
            nu = T(1) / T(4) * hu;
            nv = T(1) / T(2) * hv;
        } else {                 // row 2 J: completes J - 1
            su += T(1) / T(4) * hu;
            if (coarse && J > J0 && J <= J1) {
                const int k = cg.idx(I, J - 1);
                const unsigned m = __ldg(C.o.mask + k);
                V2 b;
                b.x = (m & U_IDENTITY) ? T(0) : su;
                b.y = (m & V_IDENTITY) ? T(0) : sv;
                C.b[k] = b;
            }
            su = nu + (!g.py && J == 0 ? T(1) : T(3) / T(4)) * hu;
            sv = nv + hv;
        }
        col.template fetch<false>(old, j + 3, nullptr);   // its slot is free now
    };
    for (int j = ja; j <= jb; j += 4) {
        step(j, ring[3], ring[0], ring[1]);
        if (j + 1 > jb) break;
        step(j + 1, ring[0], ring[1], ring[2]);
        if (j + 2 > jb) break;
        step(j + 2, ring[1], ring[2], ring[3]);
        if (j + 3 > jb) break;
        step(j + 3, ring[2], ring[3], ring[0]);
    }
}

// The prolongation (prolonged) and two sweeps: xout = two sweeps of x2 + P xc.  Only for levels halved in both directions.
// DOT: also the r.z of the conjugate-gradient step, z being xout 2^r32_exp (the finest level's way up).  A pass of its own
// for it cost 5.5 us at 320 x 160 and 10 us at 2560 x 320; here a row's r is read a row ahead, and four blocks an SM are
// kept (three rows ahead took 148 registers, three blocks, and a second wave: 2560 x 320 went from 192 to 202 us a step
// instead of to 189).
template <typename T, bool UNI, bool DOT>
__global__ void __launch_bounds__(32 * VCYCLE_WARPS, UNI ? 4 : 3) k_vcycle_up(LevelView<T> L, LevelView<T> C, const typename Vec2<T>::type* __restrict__ x2,
                                                                const typename Vec2<T>::type* __restrict__ xc,
                                                                typename Vec2<T>::type* __restrict__ xout, int rows, const int* done, CGDot dot) {
    NK_BATCH_ENTER(L.o.g, L, C, x2, xc, xout, done, dot)
    if (done && *(volatile const int*)done) return;
    using V2 = typename Vec2<T>::type;
    using Row = typename LevelColumn<T>::Row;
    const DevGrid<T>&g = L.o.g, &cg = C.o.g;
    const int lane = threadIdx.x;
    const int strip = blockIdx.x * VCYCLE_WARPS + threadIdx.y;
    const int j0 = blockIdx.y * rows, j1 = j0 + rows < g.Ny ? j0 + rows : g.Ny;
    const bool active = strip * UP_COLS < g.Nx;   // whole warp
    if (!DOT && !active) return;
    double rz[1] = {0.0};
    const int ze = DOT ? dot.sc->r32_exp : 0;
    if (active) {
    const int i = strip * UP_COLS - UP_FIRST + lane;
    const LevelColumn<T> col(L, i);
    const bool own = lane >= UP_FIRST && lane < UP_FIRST + UP_COLS && i < g.Nx;
    V2* const xw = own ? xout + i : nullptr;
    // coarse columns I and Ic (the second parent); beyond a Bounded edge the centre-located parent is the edge's and the
    // face-located one the wall's zero.  The coarse iterate is zero on its identity rows.
    const int is = col.iw < g.Nx ? col.iw : g.Nx - 1;   // the wall column takes no correction (it is inactive)
    const bool ei = (is & 1) == 0;
    const int I = is >> 1, Iq = ei ? I - 1 : I + 1;
    const bool ic_in = cg.px || (Iq >= 0 && Iq < cg.Nx);
    const int Ic = cg.px ? wrapn(Iq, cg.Nx) : (Iq < 0 ? 0 : (Iq > cg.Nx - 1 ? cg.Nx - 1 : Iq));
    const T fa = ei ? T(1) : T(1) / T(2), fb = ei || !ic_in ? T(0) : T(1) / T(2);
    struct Fine { Row r; V2 a0, a1, b0, b1; };          // a row and the coarse pairs (I, Ic) of its two parent rows
    auto fetch = [&](Fine& f, int j) {
        col.template fetch<true>(f.r, j, x2);
        int js = col.row(j);
        js = js < g.Ny ? js : g.Ny - 1;
        const int J = js >> 1, Jq = (js & 1) == 0 ? J - 1 : J + 1;
        const int Jc = cg.py ? (Jq < 0 ? cg.Ny - 1 : (Jq >= cg.Ny ? 0 : Jq)) : (Jq < 0 ? 0 : (Jq > cg.Ny - 1 ? cg.Ny - 1 : Jq));
        const V2 *p = xc + J * cg.pitch, *q = xc + Jc * cg.pitch;
        f.a0 = p[I];
        f.a1 = p[Ic];
        f.b0 = q[I];
        f.b1 = q[Ic];
    };
    auto settle = [&](Fine& f, int j) {                 // x + P xc once the reads have arrived
        Row& r = f.r;
        col.template settle<UNI, true>(r, j);
        const int js = col.row(j);
        const bool ej = (js & 1) == 0;
        const T ga = ej ? T(1) : T(1) / T(2), gb = ej || (!cg.py && (js >> 1) + 1 >= cg.Ny) ? T(0) : T(1) / T(2);
        const T au = fa * f.a0.x + fb * f.a1.x, bu = fa * f.b0.x + fb * f.b1.x;
        const T av = T(3) / T(4) * f.a0.y + T(1) / T(4) * f.a1.y, bv = T(3) / T(4) * f.b0.y + T(1) / T(4) * f.b1.y;
        if (!(r.m & U_IDENTITY)) r.x.x += T(3) / T(4) * au + T(1) / T(4) * bu;
        if (!(r.m & V_IDENTITY)) r.x.y += ga * av + gb * bv;
    };
    Stage<T, UNI> s1(g, col.iw), s2(g, col.iw);
    const int ja = j0 - 2, jb = j1;
    Fine ring[4];
    V2 y;                                               // the first sweep at row j - 1, then at row j
    double2 res = make_double2(0.0, 0.0);               // r at row j - 1
    const double2* const rr = DOT ? dot.r + (own ? i : 0) : nullptr;
    fetch(ring[0], ja);
    fetch(ring[1], ja + 1);
    fetch(ring[2], ja + 2);
    settle(ring[0], ja);
    ring[3] = ring[0];
    s1.mu = active_u<T>(ring[0].r, ring[0].r.x.x);
    s1.mv = active_v<T>(ring[0].r, ring[0].r.x.y);
    y.x = y.y = T(0);
    auto step = [&](int j, Fine& fo, Fine& fc, Fine& fn) {
        settle(fn, j + 1);
        const Row &old = fo.r, &cur = fc.r, &nxt = fn.r;
        T du, dv;
        s1.push(UNI ? 0 : col.row(j), UNI ? 0 : col.face(j), active_u<T>(nxt, nxt.x.x), active_v<T>(nxt, nxt.x.y), cur.c.x, nxt.c.y, du, dv);
        const V2 prev = y;
        y.x = cur.x.x + (cur.b.x - (cur.c.z * cur.x.x - du)) * cur.w.x;
        y.y = cur.x.y + (cur.b.y - (cur.c.w * cur.x.y - dv)) * cur.w.y;
        T eu, ev;                                       // the second sweep at row j - 1
        s2.push(UNI ? 0 : col.row(j - 1), UNI ? 0 : col.face(j - 1), active_u<T>(cur, y.x), active_v<T>(cur, y.y), old.c.x, cur.c.y, eu, ev);
        if (xw && j > j0 && j <= j1) {
            V2 o;
            o.x = prev.x + (old.b.x - (old.c.z * prev.x - eu)) * old.w.x;
            o.y = prev.y + (old.b.y - (old.c.w * prev.y - ev)) * old.w.y;
            xw[(j - 1) * g.pitch] = o;
            if (DOT) rz[0] = fma(res.x, widen_pow2(o.x, ze), fma(res.y, widen_pow2(o.y, ze), rz[0]));
        }
        if (DOT && j >= j0) res = rr[min(j, j1 - 1) * g.pitch];   // a row ahead
        fetch(fo, j + 3);
    };
    for (int j = ja; j <= jb; j += 4) {
        step(j, ring[3], ring[0], ring[1]);
        if (j + 1 > jb) break;
        step(j + 1, ring[0], ring[1], ring[2]);
        if (j + 2 > jb) break;
        step(j + 2, ring[1], ring[2], ring[3]);
        if (j + 3 > jb) break;
        step(j + 3, ring[2], ring[3], ring[0]);
    }
    }
    if constexpr (DOT) {
        const CGDotScalars scalars(dot.sc);
        if (grid_sum<1>(rz, dot.partials, &dot.sc->ticket) && threadIdx.x == 0 && threadIdx.y == 0) scalars.finish(dot, rz[0]);
    }
}

// Rows a walk writes: as long as leaves every SM about sixteen walks (2560 x 320 solve 13.2 ms, 14.2 with eight and 13.4
// with twenty-four), at least enough that the rows above it are not most of its work.
static int vcycle_rows(int strips, int ny, int least) {
    int r = (int)(((long long)strips * ny + 16 * SM_COUNT - 1) / (16 * SM_COUNT));
    return r < least ? least : (r > 32 ? 32 : r);
}

template <typename T>
void launch_vcycle_down(const LevelView<T>& L, const LevelView<T>& C, typename Vec2<T>::type* x2, const int* done, cudaStream_t s) {
    const int strips = (L.o.g.Nx + DOWN_COLS - 1) / DOWN_COLS, rows = vcycle_rows(strips, C.o.g.Ny, 2);
    dim3 block(32, VCYCLE_WARPS), grid((strips + VCYCLE_WARPS - 1) / VCYCLE_WARPS, (C.o.g.Ny + rows - 1) / rows, batch_slots());
    if (L.o.g.h != T(0)) k_vcycle_down<T, true><<<grid, block, 0, s>>>(L, C, x2, rows, done);
    else k_vcycle_down<T, false><<<grid, block, 0, s>>>(L, C, x2, rows, done);
    count_launch();
}
static dim3 vcycle_up_grid(int Nx, int Ny, int& rows) {
    const int strips = (Nx + UP_COLS - 1) / UP_COLS;
    rows = vcycle_rows(strips, Ny, 4);
    return dim3((strips + VCYCLE_WARPS - 1) / VCYCLE_WARPS, (Ny + rows - 1) / rows);
}
size_t vcycle_up_blocks(int Nx, int Ny) {
    int rows;
    const dim3 grid = vcycle_up_grid(Nx, Ny, rows);
    return (size_t)grid.x * grid.y;
}
template <typename T>
void launch_vcycle_up(const LevelView<T>& L, const LevelView<T>& C, const typename Vec2<T>::type* x2, const typename Vec2<T>::type* xc,
                      typename Vec2<T>::type* xout, const int* done, const CGDot* dot, cudaStream_t s) {
    int rows;
    dim3 block(32, VCYCLE_WARPS), grid = vcycle_up_grid(L.o.g.Nx, L.o.g.Ny, rows);
    grid.z = batch_slots();
    const bool uni = L.o.g.h != T(0);
    if (dot && uni) k_vcycle_up<T, true, true><<<grid, block, 0, s>>>(L, C, x2, xc, xout, rows, done, *dot);
    else if (dot) k_vcycle_up<T, false, true><<<grid, block, 0, s>>>(L, C, x2, xc, xout, rows, done, *dot);
    else if (uni) k_vcycle_up<T, true, false><<<grid, block, 0, s>>>(L, C, x2, xc, xout, rows, done, CGDot{});
    else k_vcycle_up<T, false, false><<<grid, block, 0, s>>>(L, C, x2, xc, xout, rows, done, CGDot{});
    count_launch();
}
template void launch_vcycle_down<float>(const LevelView<float>&, const LevelView<float>&, float2*, const int*, cudaStream_t);
template void launch_vcycle_up<float>(const LevelView<float>&, const LevelView<float>&, const float2*, const float2*, float2*, const int*,
                                      const CGDot*, cudaStream_t);

}  // namespace nk
