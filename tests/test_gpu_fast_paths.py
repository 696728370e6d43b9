"""The kernels' fast paths against the oracle at the sizes and values where they hand over to the general path."""
import numpy as np
import pytest

import nunatak_gb300 as nk

gpu = pytest.mark.gpu


# The grounded fraction, the face fractions, the effective pressure and the ice mask skip their divisions away from the
# grounding line and the margin.  Flotations of exactly zero, of one rounding, and of each sign next to the other, and
# thicknesses at both ends of the mask's transition, take both paths.  Both backends evaluate H + (ρw / ρi) b in FP64:
# one rounding of a flotation of 1e3 m is 1e-13 m, so fractions of flotations of 1 m and more agree to 1e-12, and the
# planted zeros (H = 0 over b = 0) are exact on both.
@gpu
@pytest.mark.parametrize("nx, ny, topology", [(33, 9, ("Bounded", "Bounded")), (32, 8, ("Periodic", "Bounded")), (5, 40, ("Bounded", "Periodic")),
                                              (64, 17, ("Periodic", "Periodic"))])
def test_geometry_at_the_grounding_line_and_the_margin(oracle_cls, gpu_cls, nx, ny, topology):
    rng = np.random.default_rng(nx * 100 + ny)
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 1e3), y=(0.0, ny * 1e3), topology=topology)
    desc = nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                               grounding=nk.SubgridGroundedFraction(), masking=nk.SmoothIceMask(minimum_thickness=2.0, transition_thickness=3.0))
    H = 500.0 + 300.0 * rng.standard_normal((ny, nx))
    bed = np.where(rng.random((ny, nx)) < 0.5, -900.0, 100.0) + 50.0 * rng.standard_normal((ny, nx))
    bed[:, : nx // 3] = 200.0       # a grounded and a floating region around the mixed one
    bed[:, 2 * nx // 3:] = -2000.0
    H = np.clip(H, 50.0, None)
    for value in (0.0, 2.0, 5.0, 2.0 + 1e-12, 5.0 - 1e-12, 3.5, 1e-300):
        H[rng.integers(ny, size=3), rng.integers(nx, size=3)] = value
    zero = rng.random((ny, nx)) < 0.05
    H[zero], bed[zero] = 0.0, 0.0
    got, want = [], []
    for cls, out in ((gpu_cls, got), (oracle_cls, want)):
        P = cls(grid, desc)
        P.set("H", H)
        P.set("bed", bed)
        P.compute_geometry()
        out += [P.get(n) for n in ("phi", "phi_u", "phi_v", "N", "ice_mask", "s")]
        P.close()
    for g, w in zip(got, want):
        assert np.max(np.abs(g - w)) <= 1e-12 * max(1.0, np.max(np.abs(w)))
    assert 0 < np.mean(want[0] == 1.0) < 1 and np.any(want[0] == 0.0)


# The coarse levels' cluster kernel (all levels from the first of at most 16384 cells, in FP32 and in FP64) against the
# oracle's V-cycle: one CTA and many, rows that do not divide by the CTAs, CTAs without rows, axes that stop halving
# before the other, periodic seams inside and across CTAs, odd and even sweep counts, no coarse level at all, and a top
# level one row beyond the limit.  FP64: the sums of products against the oracle's differences round at 1e-16 of
# rowsum |x| in each of the ~50 sweeps, so 1e-12 of the largest entry; FP32: the same with 6e-8, so 1e-4.
@gpu
@pytest.mark.parametrize("precision, tol", [("fp64", 1e-12), ("mixed", 1e-4)])
@pytest.mark.parametrize("nx, ny, topology, sweeps, coarsest, minimum", [
    (16, 16, ("Bounded", "Bounded"), 2, 20, 4),
    (64, 34, ("Bounded", "Bounded"), 2, 20, 16),
    (96, 40, ("Periodic", "Bounded"), 1, 7, 2),
    (40, 96, ("Bounded", "Periodic"), 3, 6, 4),
    (72, 48, ("Periodic", "Periodic"), 2, 1, 3),
    (75, 45, ("Bounded", "Bounded"), 2, 20, 4),
    (128, 128, ("Bounded", "Bounded"), 2, 20, 32),
    (128, 130, ("Bounded", "Bounded"), 2, 20, 32),
    (512, 18, ("Bounded", "Bounded"), 2, 5, 9),
])
def test_coarse_levels_in_a_cluster(oracle_cls, gpu_cls, nx, ny, topology, sweeps, coarsest, minimum, precision, tol):
    rng = np.random.default_rng(nx + ny)
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 2e3), y=(0.0, ny * 1.5e3), topology=topology)
    mg = nk.StressBalanceMultigridPreconditioner(smoothing_sweeps=sweeps, coarsest_sweeps=coarsest, minimum_coarse_size=minimum)

    def vcycle(cls, precision):
        solver = nk.StressBalanceSolver(preconditioner=mg, precision=precision)
        P = cls(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                          stress_balance=nk.DepthIntegrated(side_walls=nk.NoSlipWalls()), velocity_solver=solver))
        H = np.clip(1000.0 + 400.0 * np.random.default_rng(1).standard_normal((ny, nx)), 0.0, None)
        H[:, : nx // 8] = 0.0   # ice free: identity rows
        for n, a in (("H", H), ("bed", 10.0), ("C", 1e9), ("A", 3e-24)):
            P.set(n, a)
        P.compute_geometry()
        r = np.random.default_rng(2)
        P.set("u", 1e-5 * r.standard_normal(P.shape("u")))
        P.set("v", 1e-5 * r.standard_normal(P.shape("v")))
        P.update_coefficients()
        z = P.precondition(ru, rv)
        P.close()
        return z

    fx, fy = grid.face_count(0), grid.face_count(1)
    ru, rv = 1e10 * rng.standard_normal((ny, fx)), 1e10 * rng.standard_normal((fy, nx))
    got, want = vcycle(gpu_cls, precision), vcycle(oracle_cls, "fp64")
    for g, w in zip(got, want):
        g, w = g[:ny, :nx], w[:ny, :nx]
        assert np.max(np.abs(g - w)) <= tol * np.max(np.abs(w))


# The coarsest level's sweeps with several halo rows (FP32, clusters of more than one CTA): sweep counts that end on an
# exchange, one after it and before the first, windows that wrap round a periodic axis and that reach both walls, CTAs
# without rows, no finer level.  Tolerance as above.
@gpu
@pytest.mark.parametrize("coarsest", [4, 9, 17, 20])
@pytest.mark.parametrize("nx, ny, topology, minimum", [
    (64, 64, ("Periodic", "Periodic"), 16),
    (160, 80, ("Bounded", "Bounded"), 20),
    (64, 48, ("Bounded", "Periodic"), 3),
    (60, 44, ("Periodic", "Bounded"), 44),
])
def test_coarsest_sweeps_with_a_halo(oracle_cls, gpu_cls, nx, ny, topology, minimum, coarsest):
    rng = np.random.default_rng(nx + ny)
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 2e3), y=(0.0, ny * 1.5e3), topology=topology)
    mg = nk.StressBalanceMultigridPreconditioner(coarsest_sweeps=coarsest, minimum_coarse_size=minimum)
    H = np.clip(1000.0 + 400.0 * rng.standard_normal((ny, nx)), 0.0, None)
    H[:, : nx // 8] = 0.0
    ru, rv = 1e10 * rng.standard_normal((ny, grid.face_count(0))), 1e10 * rng.standard_normal((grid.face_count(1), nx))
    z = []
    for cls, precision in ((gpu_cls, "mixed"), (oracle_cls, "fp64")):
        P = cls(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                          stress_balance=nk.DepthIntegrated(side_walls=nk.NoSlipWalls()),
                                          velocity_solver=nk.StressBalanceSolver(preconditioner=mg, precision=precision)))
        for n, a in (("H", H), ("bed", 10.0), ("C", 1e9), ("A", 3e-24)):
            P.set(n, a)
        P.compute_geometry()
        P.update_coefficients()
        z.append([a[:ny, :nx] for a in P.precondition(ru, rv)])
        P.close()
    for g, w in zip(*z):
        assert np.max(np.abs(g - w)) <= 1e-4 * np.max(np.abs(w))


# One pass down and one up a level (FP32 levels above the cluster's 16384 cells, two sweeps, both axes halved): widths at
# and beside multiples of the 26 and 28 columns that a warp writes, rows that do not divide by a walk, one and two such
# levels, periodic seams, faces that are not square, walls with shear, ice-free cells.  Tolerance as above.
@gpu
@pytest.mark.parametrize("nx, ny, topology, stretch", [
    (260, 66, ("Bounded", "Bounded"), 1.0),
    (280, 62, ("Periodic", "Bounded"), 1.0),
    (262, 90, ("Bounded", "Periodic"), 1.5),
    (150, 130, ("Periodic", "Periodic"), 1.0),
    (364, 210, ("Bounded", "Bounded"), 0.7),
    (416, 224, ("Bounded", "Bounded"), 1.0),
])
def test_vcycle_halves(oracle_cls, gpu_cls, nx, ny, topology, stretch):
    rng = np.random.default_rng(nx + ny)
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 2e3), y=(0.0, ny * 2e3 * stretch), topology=topology)
    mg = nk.StressBalanceMultigridPreconditioner(minimum_coarse_size=20)
    H = np.clip(1000.0 + 400.0 * np.random.default_rng(1).standard_normal((ny, nx)), 0.0, None)
    H[:, : nx // 8] = 0.0
    H[ny // 2, :] = 0.0
    ru, rv = 1e10 * rng.standard_normal((ny, grid.face_count(0))), 1e10 * rng.standard_normal((grid.face_count(1), nx))
    z = []
    for cls, precision in ((gpu_cls, "mixed"), (oracle_cls, "fp64")):
        P = cls(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                          stress_balance=nk.DepthIntegrated(side_walls=nk.NoSlipWalls()),
                                          velocity_solver=nk.StressBalanceSolver(preconditioner=mg, precision=precision)))
        for n, a in (("H", H), ("bed", 10.0), ("C", 1e9), ("A", 3e-24)):
            P.set(n, a)
        P.compute_geometry()
        r = np.random.default_rng(2)
        P.set("u", 1e-5 * r.standard_normal(P.shape("u")))
        P.set("v", 1e-5 * r.standard_normal(P.shape("v")))
        P.update_coefficients()
        z.append(P.precondition(ru, rv))
        P.close()
    for g, w in zip(*z):
        g, w = g[:ny, :nx], w[:ny, :nx]
        assert np.max(np.abs(g - w)) <= 1e-4 * np.max(np.abs(w))


# The conjugate-gradient kernels at the sizes where their launch shapes change: one row a walk (up to 8 strip rows an SM),
# two rows, long walks (more than 20 strip rows an SM) with a remainder of rows, blocks of 1, 2 and more warps, widths of
# 30 k and 32 k columns and one beside, a periodic seam, faces that are not square.  Ten steps from rest against the
# oracle's: the operator's sums round at 1e-16 of their terms, ten steps carry that to 1e-12 of the largest velocity.
@gpu
@pytest.mark.parametrize("nx, ny, topology, stretch", [
    (30, 9, ("Bounded", "Bounded"), 1.0),
    (33, 40, ("Periodic", "Bounded"), 1.0),
    (61, 64, ("Bounded", "Periodic"), 1.0),
    (128, 61, ("Bounded", "Bounded"), 1.25),
    (301, 131, ("Bounded", "Bounded"), 1.0),
    (420, 215, ("Periodic", "Periodic"), 1.0),
    (481, 203, ("Bounded", "Bounded"), 1.0),
    (513, 190, ("Periodic", "Bounded"), 0.8),
])
def test_cg_steps_at_the_launch_shapes_edges(oracle_cls, gpu_cls, nx, ny, topology, stretch):
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 2e3), y=(0.0, ny * 2e3 * stretch), topology=topology)
    solver = nk.StressBalanceSolver(linear_iteration_control=nk.FixedIterations(10), picard_iteration_control=nk.FixedIterations(1))
    desc = nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                               stress_balance=nk.DepthIntegrated(side_walls=nk.NoSlipWalls()), velocity_solver=solver)
    H = np.clip(1000.0 + 300.0 * np.random.default_rng(nx).standard_normal((ny, nx)), 0.0, None)
    H[ny // 3: ny // 3 + 2] = 0.0
    out = []
    for cls in (gpu_cls, oracle_cls):
        P = cls(grid, desc)
        for n, a in (("H", H), ("bed", 10.0), ("C", 1e9), ("A", 3e-24)):
            P.set(n, a)
        P.compute_geometry()
        st = P.picard_solve()
        out.append((P.get("u"), P.get("v")))
        assert st.linear_iterations_total == 10
        P.close()
    for g, w in zip(*out):
        assert np.max(np.abs(g - w)) <= 1e-12 * np.max(np.abs(w))


# The r.z of a preconditioned step is taken by the kernel that ends the V-cycle: one cluster (60 x 40), the FP32 way up
# with both metrics (200 x 150) and with more blocks than the grid has 2-D tiles (24 x 5000), and a pass of its own after
# the grid-wide FP64 levels.  Three steps from rest against the oracle's: an FP64 V-cycle agrees to 1e-12 of its largest
# value, and three steps' quotients leave that below 1e-9; an FP32 one to 1e-4, below 1e-3.
@gpu
@pytest.mark.parametrize("precision, tol", [("fp64", 1e-9), ("mixed", 1e-3)])
@pytest.mark.parametrize("nx, ny, topology, stretch", [
    (60, 40, ("Bounded", "Bounded"), 1.0),
    (200, 150, ("Periodic", "Bounded"), 1.0),
    (200, 150, ("Bounded", "Bounded"), 1.25),
    (24, 5000, ("Bounded", "Periodic"), 1.0),
])
def test_preconditioned_steps(oracle_cls, gpu_cls, nx, ny, topology, stretch, precision, tol):
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 2e3), y=(0.0, ny * 2e3 * stretch), topology=topology)
    H = np.clip(1000.0 + 300.0 * np.random.default_rng(nx).standard_normal((ny, nx)), 100.0, None)
    out = []
    for cls, p in ((gpu_cls, precision), (oracle_cls, "fp64")):
        solver = nk.StressBalanceSolver(linear_iteration_control=nk.FixedIterations(3), picard_iteration_control=nk.FixedIterations(1),
                                        preconditioner=nk.StressBalanceMultigridPreconditioner(minimum_coarse_size=8), precision=p)
        P = cls(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                          stress_balance=nk.DepthIntegrated(side_walls=nk.NoSlipWalls()), velocity_solver=solver))
        for n, a in (("H", H), ("bed", 10.0), ("C", 1e9), ("A", 3e-24)):
            P.set(n, a)
        P.compute_geometry()
        assert P.picard_solve().linear_iterations_total == 3
        out.append((P.get("u"), P.get("v")))
        P.close()
    for g, w in zip(*out):
        assert np.max(np.abs(g - w)) <= tol * np.max(np.abs(w))


# Conjugate gradients in one cluster: fewer rows than CTAs, several rows a CTA with a shorter last one, a full row of
# threads (512 columns) and one column more (the grid-wide kernels), both seams, with the Jacobi preconditioner and without.
# Ten steps against the oracle's as above (1e-12), and one solve to convergence in the oracle's number of steps.
@gpu
@pytest.mark.parametrize("preconditioner", [nk.StressBalanceDiagonalPreconditioner(), None])
@pytest.mark.parametrize("nx, ny, topology", [
    (4, 4, ("Periodic", "Periodic")),
    (5, 33, ("Bounded", "Periodic")),
    (9, 300, ("Periodic", "Bounded")),
    (64, 128, ("Bounded", "Bounded")),
    (512, 16, ("Bounded", "Bounded")),
    (513, 16, ("Periodic", "Bounded")),
])
def test_cg_in_a_cluster(oracle_cls, gpu_cls, nx, ny, topology, preconditioner):
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 2e3), y=(0.0, ny * 2e3), topology=topology)
    H = np.clip(1000.0 + 300.0 * np.random.default_rng(nx).standard_normal((ny, nx)), 0.0, None)
    H[ny // 3] = 0.0
    for control, tol in ((nk.FixedIterations(10), 1e-12), (nk.Convergence(reltol=1e-3, maxiter=3000), 1e-6)):
        solver = nk.StressBalanceSolver(linear_iteration_control=control, picard_iteration_control=nk.FixedIterations(1),
                                        preconditioner=preconditioner)
        out = []
        for cls in (gpu_cls, oracle_cls):
            P = cls(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                              stress_balance=nk.DepthIntegrated(side_walls=nk.NoSlipWalls()), velocity_solver=solver))
            for n, a in (("H", H), ("bed", 10.0), ("C", 1e9), ("A", 3e-24)):
                P.set(n, a)
            P.compute_geometry()
            st = P.picard_solve()
            out.append((P.get("u"), P.get("v"), st.linear_iterations_total, st.status))
            P.close()
        assert out[0][2:] == out[1][2:]
        for g, w in zip(out[0][:2], out[1][:2]):
            assert np.max(np.abs(g - w)) <= tol * np.max(np.abs(w))


# Axes of unequal spacing: at a wall the face spacing (the edge cell's own width) is not that of the next face, and with
# no-slip walls the corners on the wall enter the rows beside it.  Ten steps against the oracle's as above (1e-12), and an
# FP32 V-cycle against its FP64 one (1e-4).
@gpu
@pytest.mark.parametrize("nx, ny, topology", [(70, 61, ("Bounded", "Bounded")), (160, 150, ("Bounded", "Bounded")), (160, 150, ("Periodic", "Periodic"))])
def test_unequal_spacing_at_the_walls(oracle_cls, gpu_cls, nx, ny, topology):
    rng = np.random.default_rng(nx)
    faces = [np.concatenate([[0.0], np.cumsum(rng.uniform(1e3, 3e3, n))]).tolist() for n in (nx, ny)]
    grid = nk.RectilinearGrid(size=(nx, ny), x=faces[0], y=faces[1], topology=topology)
    H = np.clip(1000.0 + 300.0 * rng.standard_normal((ny, nx)), 100.0, None)
    ru, rv = 1e10 * rng.standard_normal((ny, grid.face_count(0))), 1e10 * rng.standard_normal((grid.face_count(1), nx))
    for kw, tol in ((dict(), 1e-12), (dict(preconditioner=nk.StressBalanceMultigridPreconditioner(minimum_coarse_size=20)), 1e-4)):
        out = []
        for cls in (gpu_cls, oracle_cls):
            mixed = {"precision": "mixed"} if kw and cls is gpu_cls else {}
            solver = nk.StressBalanceSolver(linear_iteration_control=nk.FixedIterations(10),
                                            picard_iteration_control=nk.FixedIterations(1), **kw, **mixed)
            P = cls(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                              stress_balance=nk.DepthIntegrated(side_walls=nk.NoSlipWalls()), velocity_solver=solver))
            for n, a in (("H", H), ("bed", 10.0), ("C", 1e9), ("A", 3e-24)):
                P.set(n, a)
            P.compute_geometry()
            if kw:
                P.update_coefficients()
                out.append([a[:ny, :nx] for a in P.precondition(ru, rv)])
            else:
                P.picard_solve()
                out.append([P.get("u"), P.get("v")])
            P.close()
        for g, w in zip(*out):
            assert np.max(np.abs(g - w)) <= tol * np.max(np.abs(w))


# The FP64 <-> FP32 conversions on the integer units are the hardware conversions' bits, so a mixed solve keeps its
# residuals' scale: right-hand sides far outside the FP32 range (2^-400 to 2^400, whose squared norms FP64 still holds)
# converge in the same steps, to the same digits, as those near one.
@gpu
@pytest.mark.parametrize("exponent", [-400, -300, 300, 400])
def test_mixed_solve_scales_with_its_right_hand_side(gpu_cls, exponent):
    nx, ny = 64, 40
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 2e3), y=(0.0, ny * 2e3))
    solver = nk.StressBalanceSolver(linear_iteration_control=nk.Convergence(reltol=1e-12, maxiter=200), precision="mixed",
                                    preconditioner=nk.StressBalanceMultigridPreconditioner(minimum_coarse_size=8))
    P = gpu_cls(grid, nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                                          velocity_solver=solver))
    for n, a in (("H", 1000.0), ("bed", 10.0), ("C", 1e9), ("A", 3e-24), ("u", 1e-6), ("v", 0.0)):
        P.set(n, a)
    P.compute_geometry()
    P.update_coefficients()
    rng = np.random.default_rng(5)
    bu, bv = rng.standard_normal(P.shape("u")), rng.standard_normal(P.shape("v"))
    res = []
    for scale in (1.0, 2.0 ** exponent):
        P.set("u", 0.0)
        P.set("v", 0.0)
        st = P.linear_solve(bu * scale, bv * scale)
        res.append((P.get("u") / scale, P.get("v") / scale, st.linear_iterations_total, st.status))
    P.close()
    assert res[0][2:] == res[1][2:]
    for a, b in zip(res[0][:2], res[1][:2]):
        assert np.array_equal(a, b)


# The thickness stages with each cell's WENO reconstructions and limiter in one kernel: axes shorter and longer than a
# stencil's wrap, widths beside 32, both periodic seams, no bounds, bounds out of reach (no division) and bounds that the
# reconstructions pass (the limiter divides), an ice-free margin.  Reconstructions round at 1e-16 of the thickness, the
# shared denominators at a few more; three stages carry that to 1e-12 of the largest thickness.
@gpu
@pytest.mark.parametrize("bounds", [None, (0.0, 1e5), (200.0, 900.0)])
@pytest.mark.parametrize("nx, ny, topology", [(5, 7, ("Periodic", "Periodic")), (33, 9, ("Bounded", "Periodic")), (31, 40, ("Periodic", "Bounded")),
                                              (64, 33, ("Bounded", "Bounded"))])
def test_weno_faces_and_limiter(oracle_cls, gpu_cls, nx, ny, topology, bounds):
    rng = np.random.default_rng(nx + 7 * ny)
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 1e3), y=(0.0, ny * 1.3e3), topology=topology, halo=(4, 4))
    desc = nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(),
                               grounding=nk.SubgridGroundedFraction())
    H = 550.0 + 340.0 * np.tanh(rng.standard_normal((ny, nx)))
    if bounds != (200.0, 900.0):
        H[: max(1, ny // 4), : max(1, nx // 4)] = 0.0
    out = []
    for cls in (gpu_cls, oracle_cls):
        P = cls(grid, desc)
        r = np.random.default_rng(3)
        P.set("H", H)
        P.set("bed", -450.0)
        P.set("u", 1e-5 * r.standard_normal(P.shape("u")))
        P.set("v", 1e-5 * r.standard_normal(P.shape("v")))
        P.energy_set("surface_mass_balance", 1e-8)
        P.energy_set("basal_melt_rate", 2e-8)
        P.set_thickness_advection(nk.WENO(order=5, bounds=bounds))
        P.compute_geometry()
        P.step_thickness(5e6)
        out.append([P.get(n) for n in ("H", "tau_u", "tau_v")] + [P.energy_get("clipped_thickness")])
        P.close()
    for g, w in zip(*out):
        assert np.max(np.abs(g - w)) <= 1e-12 * max(np.max(np.abs(w)), 1.0)


# The reverse of a stage on axes where a stencil reaches past both edges, reads a cell twice or only just wraps: the
# gradient of a weighted sum of the thickness after two steps against centred differences of the steps themselves.  One
# FP64 step's rounding over the difference 2 x 1e-3 m leaves 1e-9 of a weight; the difference's own second-order error and
# the limiter's kinks are kept below by a smooth field, so 1e-6 of the largest entry.
@gpu
@pytest.mark.parametrize("scheme", [nk.WENO(order=5, bounds=(0.0, 1e5)), nk.UpwindBiased(order=3)])
@pytest.mark.parametrize("nx, ny, topology", [(4, 9, ("Periodic", "Bounded")), (5, 6, ("Periodic", "Periodic")), (9, 4, ("Bounded", "Bounded"))])
def test_stage_reverse_on_short_axes(gpu_cls, nx, ny, topology, scheme):
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 1e3), y=(0.0, ny * 1e3), topology=topology, halo=(4, 4))
    desc = nk.make_descriptors(grid, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction(), grounding=nk.SubgridGroundedFraction())
    x = (np.arange(nx)[None, :] + 0.5) / nx
    y = (np.arange(ny)[:, None] + 0.5) / ny
    H0 = 800.0 + 60.0 * np.sin(2 * np.pi * x + 0.3) + 45.0 * np.cos(2 * np.pi * y + 0.7) + 20.0 * np.sin(2 * np.pi * (x + y))
    weight = np.random.default_rng(1).random((ny, nx)) + 0.5
    r = np.random.default_rng(2)
    P = gpu_cls(grid, desc)
    P.set("bed", -300.0)
    u, v = 1e-5 * (1 + 0.3 * r.standard_normal(P.shape("u"))), 1e-5 * (-1 + 0.3 * r.standard_normal(P.shape("v")))
    P.set_thickness_advection(scheme)
    P.energy_set("surface_mass_balance", 1e-8)
    dt = 4e6

    def start(H):
        P.set("H", H)
        P.set("u", u)
        P.set("v", v)
        P.compute_geometry()

    def forward(H):
        start(H)
        for _ in range(2):
            P.step_thickness(dt)
        return P.get("H")

    start(H0)
    g = P.checkpointed_gradient(lambda step, H, *_: (float(np.sum(weight * H)), weight, None, None) if step == 2 else None, dt, 2,
                                velocity_solves=False)["H"]
    for j, i in ((0, 0), (ny - 1, nx - 1), (ny // 2, 0), (0, nx // 2), (ny // 2, nx - 1)):
        d = np.zeros_like(H0)
        d[j, i] = 1e-3
        diff = np.sum(weight * (forward(H0 + d) - forward(H0 - d))) / 2e-3
        assert abs(g[j, i] - diff) <= 1e-6 * np.max(np.abs(g))
    P.close()
