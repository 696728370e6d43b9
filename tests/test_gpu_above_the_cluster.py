"""Batches, prescribed faces and conjugate-gradient steps on grids above the cluster kernels' sizes, where the grid-wide and
the one-pass kernels run: the tests of these features at 64 x 32 run in one cluster."""
import numpy as np
import pytest

import nunatak_gb300 as nk
from nunatak_gb300 import model as M, workloads
from test_gpu_batch import alone, load
from test_inflow import YEAR, rel_l2

gpu = pytest.mark.gpu
FIXED = dict(picard_iteration_control=M.FixedIterations(2))


def solver(preconditioner, **kw):
    return M.StressBalanceSolver(preconditioner=preconditioner, linear_iteration_control=M.Convergence(reltol=1e-6, maxiter=400), **FIXED, **kw)


MG = M.StressBalanceMultigridPreconditioner(minimum_coarse_size=8)
BATCHES = {
    "one_pass_levels": (260, 66, solver(MG, precision="mixed")),          # FP32, r.z taken by the way up
    "two_one_pass_levels": (420, 220, solver(MG, precision="mixed")),
    "grid_wide_fp64_levels": (200, 150, solver(MG)),                      # r.z in a pass of its own
    "grid_wide_fp32_levels": (260, 66, solver(M.StressBalanceMultigridPreconditioner(minimum_coarse_size=8, smoothing_sweeps=3), precision="mixed")),
    "grid_wide_jacobi": (513, 16, solver(M.StressBalanceDiagonalPreconditioner())),
    "grid_wide_none": (160, 64, solver(None)),
}


# Each slot of a batch gives the bits, steps and statistics of its problem solved alone.
@gpu
@pytest.mark.parametrize("config", sorted(BATCHES))
def test_batched_slots_equal_solves_alone(config):
    nx, ny, s = BATCHES[config]
    cases = [workloads.marine_sheet(nx, ny, seed=1, seed_friction=300 + k, velocity_solver=s) for k in range(3)]
    ref = [alone(c) for c in cases]
    with nk.Batch(cases[0].grid, cases[0].descriptors(), 3) as B:
        for k, c in enumerate(cases):
            load(B, k, c)
        stats = B.picard_solve()
        for k, (u, v, st, _) in enumerate(ref):
            assert (stats[k].status, stats[k].picard_iterations, stats[k].linear_iterations_total) == \
                (st.status, st.picard_iterations, st.linear_iterations_total)
            assert stats[k].picard_change == st.picard_change and stats[k].residual_norm == st.residual_norm
            assert np.array_equal(B.problem(k).get("u"), u) and np.array_equal(B.problem(k).get("v"), v), f"slot {k}"
    assert len({st.residual_norm for _, _, st, _ in ref}) == 3 and np.any(ref[0][0] != 0.0)


# A west inflow and a prescribed segment inside the domain on a grid whose finest two levels are one-pass (mixed) or
# grid-wide (FP64): converged against the oracle, 1e-6 mixed and 1e-8 FP64 (the linear solves stop at 1e-10 of ‖r0‖, three
# Picard steps from rest on both sides; the condition of the sheet lifts that by about a hundred).
@gpu
@pytest.mark.parametrize("precision, tol", [("mixed", 1e-6), ("fp64", 1e-8)])
def test_prescribed_faces_above_the_cluster(oracle_cls, gpu_cls, precision, tol):
    nx, ny = 420, 220
    out = []
    for cls, p in ((gpu_cls, precision), (oracle_cls, "fp64")):
        s = M.StressBalanceSolver(preconditioner=MG, precision=p, linear_iteration_control=M.Convergence(reltol=1e-10, maxiter=2000),
                                  picard_iteration_control=M.FixedIterations(3))
        base = workloads.marine_sheet(nx, ny, seed=2, velocity_solver=s)
        ud = workloads.west_inflow(base.grid, 50.0).copy()
        ud[ny // 2: ny // 2 + 5, nx // 3] = 30.0 / YEAR
        P = workloads.Case("inflow", base.grid, base.config, dict(base.fields, u_prescribed=ud), dict(base.initial)).problem(cls)
        assert P.picard_solve().status == 0
        out.append((P.get("u"), P.get("v")))
        P.close()
    (u, v), (ur, vr) = out
    assert np.all(u[:, 0] == 50.0 / YEAR) and np.all(u[ny // 2: ny // 2 + 5, nx // 3] == 30.0 / YEAR)
    assert rel_l2(u, v, ur, vr) < tol


# The operator's walks just above the cluster's sizes: one row a walk with blocks of one warp (513 x 16: 288 walks) and of two
# (160 x 64: 384), two rows (301 x 131), on square cells, on others, and on unequal ones with each pair of boundaries.  Ten
# Jacobi steps from rest against the oracle's: the operator's sums round at 1e-16 of their terms, ten steps carry that to
# 1e-12 of the largest velocity.
@gpu
@pytest.mark.parametrize("stretch", [1.0, 1.25, None])
@pytest.mark.parametrize("nx, ny, topology", [(513, 16, ("Bounded", "Bounded")), (160, 64, ("Periodic", "Bounded")), (301, 131, ("Bounded", "Periodic"))])
def test_cg_steps_just_above_the_cluster(oracle_cls, gpu_cls, nx, ny, topology, stretch):
    rng = np.random.default_rng(nx)
    if stretch is None:
        x, y = (np.concatenate([[0.0], np.cumsum(rng.uniform(1e3, 3e3, n))]).tolist() for n in (nx, ny))
    else:
        x, y = (0.0, nx * 2e3), (0.0, ny * 2e3 * stretch)
    grid = nk.RectilinearGrid(size=(nx, ny), x=x, y=y, topology=topology)
    s = nk.StressBalanceSolver(linear_iteration_control=nk.FixedIterations(10), picard_iteration_control=nk.FixedIterations(1))
    H = np.clip(1000.0 + 300.0 * rng.standard_normal((ny, nx)), 0.0, None)
    H[ny // 3: ny // 3 + 2] = 0.0
    out = []
    for cls in (gpu_cls, oracle_cls):
        P = cls(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                          stress_balance=nk.DepthIntegrated(side_walls=nk.NoSlipWalls()), velocity_solver=s))
        for n, a in (("H", H), ("bed", 10.0), ("C", 1e9), ("A", 3e-24)):
            P.set(n, a)
        P.compute_geometry()
        assert P.picard_solve().linear_iterations_total == 10
        out.append((P.get("u"), P.get("v")))
        P.close()
    for g, w in zip(*out):
        assert np.max(np.abs(g - w)) <= 1e-12 * np.max(np.abs(w))
