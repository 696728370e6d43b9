"""The V-cycle's kernels where one hands over to another: short periodic axes, prescribed faces, devices without room for a
cluster, batches above the clusters' sizes, and the FP32 rows' rounding."""
import numpy as np
import pytest

import nunatak_gb300 as nk

gpu = pytest.mark.gpu


def sheet(cls, grid, solver, H):
    """An SSA sheet with no-slip walls after its first coefficient update."""
    P = cls(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                      stress_balance=nk.DepthIntegrated(side_walls=nk.NoSlipWalls()), velocity_solver=solver))
    for n, a in (("H", H), ("bed", 10.0), ("C", 1e9), ("A", 3e-24)):
        P.set(n, a)
    P.compute_geometry()
    r = np.random.default_rng(2)
    P.set("u", 1e-5 * r.standard_normal(P.shape("u")))
    P.set("v", 1e-5 * r.standard_normal(P.shape("v")))
    P.update_coefficients()
    return P


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
    ru, rv = 1e10 * rng.standard_normal((ny, grid.face_count(0))), 1e10 * rng.standard_normal((grid.face_count(1), nx))
    z = []
    for cls, precision in ((gpu_cls, "mixed"), (oracle_cls, "fp64")):
        mg = nk.StressBalanceMultigridPreconditioner(minimum_coarse_size=1)
        P = sheet(cls, grid, nk.StressBalanceSolver(preconditioner=mg, precision=precision), H)
        z.append(P.precondition(ru, rv))
        P.close()
    for g, w in zip(*z):
        g, w = g[:ny, :nx], w[:ny, :nx]
        assert np.max(np.abs(g - w)) <= 1e-4 * np.max(np.abs(w))
