"""The V-cycle's kernels where one hands over to another: short periodic axes, prescribed faces, devices without room for a
cluster, batches above the clusters' sizes, and the FP32 rows' rounding."""
import os
import subprocess
import sys

import numpy as np
import pytest

import nunatak_gb300 as nk
from nunatak_gb300 import library

gpu = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def sheet(cls, grid, solver, H, u_prescribed=None):
    """An SSA sheet with no-slip walls after its first coefficient update."""
    P = cls(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                      stress_balance=nk.DepthIntegrated(side_walls=nk.NoSlipWalls()), velocity_solver=solver))
    for n, a in (("H", H), ("bed", 10.0), ("C", 1e9), ("A", 3e-24)):
        P.set(n, a)
    if u_prescribed is not None:
        P.set("u_prescribed", u_prescribed)
    P.compute_geometry()
    r = np.random.default_rng(2)
    P.set("u", 1e-5 * r.standard_normal(P.shape("u")))
    P.set("v", 1e-5 * r.standard_normal(P.shape("v")))
    P.update_coefficients()
    return P


def residual(grid, seed):
    rng = np.random.default_rng(seed)
    return 1e10 * rng.standard_normal((grid.Ny, grid.face_count(0))), 1e10 * rng.standard_normal((grid.face_count(1), grid.Nx))


def assert_close(got, want, r, tol):
    """V-cycles of r: `tol` of the largest entry on the rows that couple, and r itself on the identity rows (walls and ice-free
    faces), whose entries are 1e19 times those and would hide them in one norm."""
    assert tol < 1e-3
    for g, w, b in zip(got, want, r):
        ny, nx = min(g.shape[0], b.shape[0]), min(g.shape[1], b.shape[1])
        g, w, b = g[:ny, :nx], w[:ny, :nx], b[:ny, :nx]
        identity = np.abs(w - b) <= 1e-7 * np.abs(b)   # (b rounded to FP32 in a mixed V-cycle)
        assert np.all(np.abs(g - b)[identity] <= 1e-7 * np.abs(b)[identity])
        assert np.max(np.abs(w[~identity])) < 1e-6 * np.max(np.abs(b))   # no identity row is left among them
        assert np.max(np.abs(g - w)[~identity]) <= tol * np.max(np.abs(w[~identity]))


def interior(grid, z):
    return [a[:grid.Ny, :grid.Nx] for a in z]


# A flowline of two, four and six rows round a periodic axis, too wide for the cluster: the one-pass kernels' walks ask for
# three rows below the grid and four above it, so only from six rows on do they take such a level.  An FP32 V-cycle against
# the oracle's FP64 one: 6e-8 of rowsum |x| in each of its ~50 sweeps, so 1e-4 of the largest entry.
@gpu
@pytest.mark.parametrize("nx, ny", [(2050, 2), (4096, 4), (4096, 8), (2050, 6)])
def test_one_pass_levels_on_a_short_periodic_axis(oracle_cls, gpu_cls, nx, ny):
    rng = np.random.default_rng(nx + ny)
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 2e3), y=(0.0, ny * 2e3), topology=("Bounded", "Periodic"), halo=(1, 1))
    H = np.clip(1000.0 + 400.0 * rng.standard_normal((ny, nx)), 0.0, None)
    H[:, : nx // 8] = 0.0
    r = residual(grid, nx)
    z = []
    for cls, precision in ((gpu_cls, "mixed"), (oracle_cls, "fp64")):
        mg = nk.StressBalanceMultigridPreconditioner(minimum_coarse_size=1)
        P = sheet(cls, grid, nk.StressBalanceSolver(preconditioner=mg, precision=precision), H)
        z.append(interior(grid, P.precondition(*r)))
        P.close()
    assert_close(z[0], z[1], interior(grid, r), 1e-4)


# One V-cycle against the oracle's: FP64 to 1e-12 and FP32 to 1e-4 of the largest entry on the rows that couple (rounding of
# 1e-16 and 6e-8 of rowsum |x| in each of its ~50 sweeps).  Faces: None for equal spacing, else the range of the cell widths.
def vcycles(gpu_cls, oracle_cls, grid, mg, precision, tol, seed):
    nx, ny = grid.Nx, grid.Ny
    H = np.clip(1000.0 + 400.0 * np.random.default_rng(seed).standard_normal((ny, nx)), 0.0, None)
    H[:, : nx // 8] = 0.0   # ice free: identity rows
    H[ny // 2, : nx // 2] = 0.0
    r = residual(grid, seed)
    z = []
    for cls, p in ((gpu_cls, precision), (oracle_cls, "fp64")):
        P = sheet(cls, grid, nk.StressBalanceSolver(preconditioner=mg, precision=p), H)
        z.append(interior(grid, P.precondition(*r)))
        P.close()
    assert_close(z[0], z[1], interior(grid, r), tol)


PRECISIONS = pytest.mark.parametrize("precision, tol", [("fp64", 1e-12), ("mixed", 1e-4)])
BB, PB, BP, PP = ("Bounded", "Bounded"), ("Periodic", "Bounded"), ("Bounded", "Periodic"), ("Periodic", "Periodic")


# The coarse levels' cluster: one CTA and many, rows that do not divide by the CTAs, CTAs without rows, axes that stop
# halving before the other, seams inside and across CTAs, odd and even sweep counts, no coarse level, FP64's largest grid
# (8192 cells, 6144 of the coarsest level) and FP32's (16384) and one row beyond, coarsest sweeps that end on, after and before an exchange of halos.
@gpu
@PRECISIONS
@pytest.mark.parametrize("nx, ny, topology, sweeps, coarsest, minimum", [
    (16, 16, BB, 2, 20, 4), (64, 34, BB, 2, 20, 16), (96, 40, PB, 1, 7, 2), (40, 96, BP, 3, 6, 4), (72, 48, PP, 2, 1, 3),
    (75, 45, BB, 2, 20, 4), (512, 16, BB, 2, 5, 8), (128, 64, PB, 2, 20, 8), (128, 128, BB, 2, 20, 32), (128, 130, BB, 2, 20, 32),
    (64, 64, PP, 2, 4, 16), (64, 64, PP, 2, 9, 16), (64, 96, BB, 2, 20, 99), (80, 80, PB, 2, 7, 99), (160, 80, BB, 2, 17, 20), (64, 48, BP, 2, 9, 3), (60, 44, PB, 2, 20, 44),
])
def test_vcycle_in_a_cluster(oracle_cls, gpu_cls, nx, ny, topology, sweeps, coarsest, minimum, precision, tol):
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 2e3), y=(0.0, ny * 1.5e3), topology=topology)
    mg = nk.StressBalanceMultigridPreconditioner(smoothing_sweeps=sweeps, coarsest_sweeps=coarsest, minimum_coarse_size=minimum)
    vcycles(gpu_cls, oracle_cls, grid, mg, precision, tol, nx + ny)


# The one-pass levels (FP32) and the grid-wide ones (FP64): widths at and beside multiples of the 26 and 28 columns of a
# warp, rows that do not divide by a walk, one and two such levels, seams, cells that are not square, unequal spacing
# with each pair of boundaries.
@gpu
@PRECISIONS
@pytest.mark.parametrize("nx, ny, topology, stretch", [
    (260, 66, BB, 1.0), (280, 62, PB, 1.0), (262, 90, BP, 1.5), (150, 130, PP, 1.0), (364, 210, BB, 0.7), (416, 224, BB, 1.0),
    (160, 150, BB, None), (160, 150, PP, None), (160, 150, PB, None), (160, 150, BP, None),
])
def test_vcycle_above_the_cluster(oracle_cls, gpu_cls, nx, ny, topology, stretch, precision, tol):
    if stretch is None:
        rng = np.random.default_rng(nx)
        x, y = (np.concatenate([[0.0], np.cumsum(rng.uniform(1e3, 3e3, n))]).tolist() for n in (nx, ny))
    else:
        x, y = (0.0, nx * 2e3), (0.0, ny * 2e3 * stretch)
    grid = nk.RectilinearGrid(size=(nx, ny), x=x, y=y, topology=topology)
    vcycles(gpu_cls, oracle_cls, grid, nk.StressBalanceMultigridPreconditioner(minimum_coarse_size=20), precision, tol, nx + ny)


# One V-cycle of a residual that does not vanish on prescribed faces: such a row keeps its part of the right-hand side in
# the residual that a level restricts, in whichever kernel the level runs.  (Conjugate gradients start from the prescribed
# values, so their residual is zero there.)
def prescribed_vcycle(nx, ny, precision):
    rng = np.random.default_rng(nx + ny)
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 2e3), y=(0.0, ny * 2e3))
    ud = np.full((ny, nx + 1), np.nan)
    ud[:, 0] = 1e-5
    ud[ny // 2, nx // 3: nx // 2] = 2e-5
    H = np.clip(1000.0 + 300.0 * rng.standard_normal((ny, nx)), 100.0, None)
    P = sheet(nk.Problem, grid, nk.StressBalanceSolver(preconditioner=nk.StressBalanceMultigridPreconditioner(minimum_coarse_size=8),
                                                       precision=precision), H, ud)
    r = residual(grid, nx)
    z = P.precondition(*r)
    P.close()
    return np.stack(interior(grid, z) + interior(grid, r))   # z, then r


def in_a_process(tmp_path, call, **env):
    """`call` (an expression over this module's names, giving an array) evaluated in a process with `env` set."""
    out = str(tmp_path / "out.npy")
    code = f"import sys; sys.path[:0] = {[ROOT, ROOT + '/nunatak.jl_gb300', ROOT + '/oracle', ROOT + '/tests']!r}\n" \
           f"import numpy as np\nfrom {__name__.rpartition('.')[2]} import *\nnp.save({out!r}, {call})\n"
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, **env), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return np.load(out)


# The coarse levels' cluster against the grid-wide launches (NK_COARSEST_SMEM=0), and the one-pass levels against the FP64
# ones, which are grid-wide at that size.  Both sides round at 1e-16 (FP32: 6e-8) of rowsum |x| in each of the ~50 sweeps.
@gpu
@pytest.mark.parametrize("precision, tol", [("fp64", 1e-12), ("mixed", 1e-4)])
def test_prescribed_faces_in_the_cluster(gpu_cls, tmp_path, precision, tol):
    got = prescribed_vcycle(40, 20, precision)
    want = in_a_process(tmp_path, f"prescribed_vcycle(40, 20, {precision!r})", NK_COARSEST_SMEM="0")
    assert_close(got[:2], want[:2], want[2:], tol)


@gpu
def test_prescribed_faces_on_one_pass_levels(gpu_cls):
    got, want = (prescribed_vcycle(260, 66, p) for p in ("mixed", "fp64"))
    assert_close(got[:2], want[:2], want[2:], 1e-4)


# The residual of a smooth iterate.  On a doubly periodic grid of one value everywhere the operator is a multiplication by the
# drag's part d = (A 1), a 750th of rowsum.  Enough sweeps (15 x 750) take an iterate to where a step no longer changes its
# last bit, a relative error of about 750 roundings; the residual b - A x must still know that error, by differences that are
# zero here, so that the coarse level corrects it.  What is left of b / d are the roundings of b, of d (the area's product and
# its product with the drag) and of the iterate: 16 of them allowed.  (A sum of products of whole values rounds the residual
# at rowsum |x|, and 750 roundings stay.)
@gpu
@pytest.mark.parametrize("precision, rounding", [("fp64", 2.0 ** -53), ("mixed", 2.0 ** -24)])
@pytest.mark.parametrize("nx, ny, dy", [(64, 64, 2e3), (128, 64, 1.5e3)])
def test_residual_of_a_smooth_iterate(gpu_cls, nx, ny, dy, precision, rounding):
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 2e3), y=(0.0, ny * dy), topology=PP)
    mg = nk.StressBalanceMultigridPreconditioner(smoothing_sweeps=12000, coarsest_sweeps=12000, minimum_coarse_size=32)
    P = gpu_cls(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                          velocity_solver=nk.StressBalanceSolver(preconditioner=mg, precision=precision)))
    for n, a in (("H", 1000.0), ("bed", 10.0), ("C", 1e8), ("A", 3e-24), ("u", 1e-5), ("v", 1e-5)):
        P.set(n, a)
    P.compute_geometry()
    P.update_coefficients()
    one = np.ones((ny, nx))
    for z, d, b in zip(P.precondition(1.7e10 * one, -0.9e10 * one), P.apply_operator(one, one), (1.7e10, -0.9e10)):
        assert np.max(np.abs(z * d / b - 1.0)) <= 16 * rounding
    P.close()


# A device without room for a cluster (NK_CLUSTERS=0): the grid-wide kernels take every solve, Jacobi on a small grid as well
# as multigrid, with the same steps and, after a fixed number of them, the same velocities.  Ten steps from rest carry the
# operator's 1e-16 to 1e-12 of the largest velocity; with FP64 V-cycles (1e-12) three quotients a step to 1e-9.
def fixed_solve(preconditioner):
    grid = nk.RectilinearGrid(size=(40, 33), x=(0.0, 80e3), y=(0.0, 66e3), topology=PB)
    solver = nk.StressBalanceSolver(linear_iteration_control=nk.FixedIterations(10), picard_iteration_control=nk.FixedIterations(1),
                                    preconditioner=preconditioner)
    P = nk.Problem(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                             velocity_solver=solver))
    H = np.clip(1000.0 + 300.0 * np.random.default_rng(3).standard_normal((33, 40)), 0.0, None)
    for n, a in (("H", H), ("bed", 10.0), ("C", 1e9), ("A", 3e-24)):
        P.set(n, a)
    P.compute_geometry()
    n0 = library.launch_count()
    st = P.picard_solve()
    out = np.concatenate([P.get("u").ravel(), P.get("v").ravel(), [st.linear_iterations_total, library.launch_count() - n0]])
    P.close()
    return out


@gpu
@pytest.mark.parametrize("preconditioner, tol", [("nk.StressBalanceDiagonalPreconditioner()", 1e-12), ("None", 1e-12),
                                                 ("nk.StressBalanceMultigridPreconditioner(minimum_coarse_size=8)", 1e-9)])
def test_without_clusters(gpu_cls, tmp_path, preconditioner, tol):
    got = fixed_solve(eval(preconditioner))
    want = in_a_process(tmp_path, f"fixed_solve({preconditioner})", NK_CLUSTERS="0")
    assert got[-2] == want[-2] == 10
    assert want[-1] - got[-1] >= 2 * 10 - 1   # in a cluster: one launch for the whole iteration, or one for a whole V-cycle
    assert np.max(np.abs(got[:-2] - want[:-2])) <= tol * np.max(np.abs(want[:-2]))
