"""Performance cases: the calls that an ice-sheet model makes of this library, over the sizes it makes them at.

A case is a dict of plain values.  `listed()` gives the named ones, `draw(rng)` one more of the same ranges,
`prepare(case, seed)` the problem, its inputs and the output buffers, `run(state)` one pass through the public entry
points, `work(case)` the bytes and operations that the pass cannot do without, and `exact(case, seed)` what the pass
returns, in plain 64-bit torch.

Fields go in from device memory (set_device) and come out to device memory (nk_problem_get_field with a device
address), the way a model that keeps its state on the GPU couples to the library; the calls whose interface is host
arrays (the adjoint, the gradient, the serving loop) are called with host arrays."""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nunatak.jl_gb300"))

import nunatak_gb300 as nk  # noqa: E402
from nunatak_gb300 import abi, library, workloads  # noqa: E402
from nunatak_gb300.server import Server  # noqa: E402

YEAR = nk.YEAR
DEV = "cuda"


def listed():
    return [
        # the smallest solve: a confined shelf, no-slip walls, Jacobi CG in FP64; bound by launches and latency
        dict(name="shelf_84x40_jacobi", kind="shelf", nx=84, ny=40),
        # one request of the serving stream at its smallest and largest size: FP32 multigrid under FP64 flexible CG
        dict(name="sheet_128x64_mixed", kind="sheet", nx=128, ny=64, precision="mixed", smoother="point"),
        dict(name="sheet_1024x512_mixed", kind="sheet", nx=1024, ny=512, precision="mixed", smoother="point"),
        # the FP64 multigrid solve, on a grid whose coarse levels are odd (150 x 90, 75 x 45)
        dict(name="sheet_300x180_fp64", kind="sheet", nx=300, ny=180, precision="fp64", smoother="point"),
        # the DIVA balance: sigma-grid rate factor, regularised Coulomb drag, a calving front
        dict(name="diva_320x160_mixed", kind="diva", nx=320, ny=160, precision="mixed"),
        # one linear solve of the scaling benchmark's ice stream from rest: Jacobi in FP64, multigrid in mixed precision
        dict(name="stream_1280x160_jacobi", kind="linear", nx=1280, ny=160, preconditioner="jacobi"),
        dict(name="stream_2560x320_mixed", kind="linear", nx=2560, ny=320, preconditioner="mixed"),
        # the reverse of a converged solve (inversion): all parameter gradients
        dict(name="adjoint_256x128_mixed", kind="adjoint", nx=256, ny=128),
        # one time step of the thickness: the default bounded WENO-5, three stages with the geometry after each
        dict(name="thickness_1500x1001_weno", kind="thickness", nx=1500, ny=1001, scheme="weno"),
        # one energy step of the columns
        dict(name="energy_700x350x10", kind="energy", nx=700, ny=350, layers=10),
        # the gradient through time steps with the velocities held: forward, re-run and reverse of every stage
        dict(name="gradient_250x125_weno", kind="gradient", nx=250, ny=125, steps=6),
        # the serving loop: requests of the four sizes in flight at once, host arrays in and out
        dict(name="serving_12", kind="serving", requests=12),
    ]


def _log_uniform(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(("shelf", "sheet", "sheet", "diva", "linear", "adjoint", "thickness", "energy", "gradient", "serving"))
    if kind == "shelf":
        nx = int(_log_uniform(rng, 82, 170))
        return dict(kind=kind, nx=nx, ny=rng.randint(20, 60))
    if kind == "sheet":
        precision = rng.choice(("mixed", "mixed", "fp64"))
        smoother = rng.choice(("point", "point", "point", "line"))
        if rng.random() < 0.3:   # an axis that does not halve
            return dict(kind=kind, nx=2 * rng.randint(40, 80) + 1, ny=rng.randint(33, 70), precision=precision, smoother="point")
        k = 2 ** rng.choice((1, 2, 3) if precision == "mixed" and smoother == "point" else (1, 2))
        return dict(kind=kind, nx=k * rng.randint(40, 88), ny=k * rng.randint(32, 44), precision=precision, smoother=smoother)
    if kind == "diva":
        k = 2 ** rng.choice((1, 2))
        return dict(kind=kind, nx=k * rng.randint(40, 70), ny=k * rng.randint(32, 40), precision=rng.choice(("mixed", "mixed", "fp64")))
    if kind == "linear":
        ny = 2 ** rng.randint(3, 5) * rng.randint(4, 9)
        return dict(kind=kind, nx=8 * ny, ny=ny, preconditioner=rng.choice(("jacobi", "mixed", "fp64")))
    if kind == "adjoint":
        return dict(kind=kind, nx=2 * rng.randint(40, 120), ny=2 * rng.randint(32, 60))
    if kind == "thickness":
        return dict(kind=kind, nx=int(_log_uniform(rng, 60, 1700)), ny=int(_log_uniform(rng, 40, 880)),
                    scheme=rng.choice(("weno", "weno", "weno unbounded", "upwind 1", "upwind 3")))
    if kind == "energy":
        return dict(kind=kind, nx=int(_log_uniform(rng, 40, 900)), ny=int(_log_uniform(rng, 30, 250)), layers=rng.randint(4, 10))
    if kind == "gradient":
        return dict(kind=kind, nx=int(_log_uniform(rng, 40, 250)), ny=int(_log_uniform(rng, 30, 120)), steps=rng.randint(2, 6))
    return dict(kind=kind, requests=rng.randint(3, 11))


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _smooth(shape, seed, cells):
    """A smooth random field (zero mean, unit deviation) of correlation length `cells`, made on the GPU."""
    g = torch.Generator().manual_seed(int(seed) & 0x7FFFFFFF)
    a = torch.randn(shape, generator=g, dtype=torch.float64).to(DEV)
    ky = torch.fft.fftfreq(shape[0], device=DEV, dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(shape[1], device=DEV, dtype=torch.float64)[None, :]
    a = torch.fft.irfft2(torch.fft.rfft2(a) * torch.exp(-2 * (math.pi * cells) ** 2 * (kx * kx + ky * ky)), s=shape)
    a = a - a.mean()
    return (a / a.std()).contiguous()


def _solver(case, **kw):
    if case.get("preconditioner") == "jacobi":
        return nk.StressBalanceSolver(preconditioner=nk.StressBalanceDiagonalPreconditioner(), **kw)
    smoother = nk.LineJacobi() if case.get("smoother") == "line" else nk.PointJacobi()
    precision = case.get("precision", case.get("preconditioner", "mixed"))
    mg = nk.StressBalanceMultigridPreconditioner(smoother=smoother, minimum_coarse_size=32)
    return nk.StressBalanceSolver(preconditioner=mg, precision=precision, **kw)


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64)).to(DEV)


def _solve_inputs(case, seed):
    """(workloads.Case without its fields, the fields on the GPU) of a whole solve."""
    nx, ny = case["nx"], case["ny"]
    if case["kind"] == "shelf":
        c = workloads.channel_shelf(nx, ny, dx=84e3 / nx)
        X = _t(c.grid.centers(0))[None, :].expand(ny, nx)
        H = torch.where(X < 80e3, 600.0 - 400.0 * X / 80e3 + 15.0 * _smooth((ny, nx), seed, nx / 20), torch.zeros_like(X))
        return c, dict(H=H.contiguous(), bed=_t(c.fields["bed"]), A=_t(c.fields["A"]))
    if case["kind"] == "diva":
        dx = 2048e3 / nx
        grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, 2048e3), y=(0.0, ny * dx), halo=(4, 4))
        X = _t(grid.centers(0))[None, :].expand(ny, nx)
        cfg = dict(Nsigma=10, stress_balance=nk.DepthIntegrated(shear=nk.DIVAShear(), side_walls=nk.FreeSlipWalls()),
                   rheology=nk.GlenFlowLaw(rate_factor="sigma", strain_rate_regularization=1e-13),
                   friction=nk.RegularizedCoulombFriction(coulomb_coefficient=0.5, exponent=1.0 / 3.0),
                   grounding=nk.SubgridGroundedFraction(), velocity_solver=_solver(case))
        bed = -100.0 - 600.0 * X / 2048e3 + 50.0 * _smooth((ny, nx), seed + 1, 80e3 / dx)
        H = torch.where(X < 1900e3, 2000.0 * torch.sqrt(torch.clamp(1.0 - (X / 1680e3) ** 2, min=0.0)), torch.zeros_like(X))
        Cf = 10.0 ** (6.5 + 0.3 * _smooth((ny, nx), seed + 2, 80e3 / dx)) * YEAR ** (1.0 / 3.0)
        z = torch.tensor([((k / 10) ** 2 + ((k + 1) / 10) ** 2) / 2 for k in range(10)], dtype=torch.float64, device=DEV)
        T = 270.0 - 17.0 * z[:, None, None] + 3.0 * _smooth((ny, nx), seed + 3, 30e3 / dx)
        return workloads.Case("diva", grid, cfg, {}), dict(H=H.contiguous(), bed=bed, C=Cf, T=T.contiguous())
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, 512e3), y=(0.0, 256e3), halo=(4, 4))
    X = _t(grid.centers(0))[None, :].expand(ny, nx)
    cells = 20e3 / (512e3 / nx)
    tight = case["kind"] == "adjoint"
    solver = _solver(case, **(dict(linear_iteration_control=nk.Convergence(reltol=1e-13, maxiter=10_000),
                                   picard_iteration_control=nk.Convergence(reltol=1e-12, maxiter=200),
                                   adjoint_iteration_control=nk.Convergence(reltol=1e-12, maxiter=400)) if tight else {}))
    cfg = dict(Nsigma=10, stress_balance=nk.DepthIntegrated(side_walls=nk.FreeSlipWalls()),
               rheology=nk.GlenFlowLaw(rate_factor=3.17e-24, strain_rate_regularization=1e-13),
               friction=nk.WeertmanFriction(exponent=1.0 / 3.0), grounding=nk.SubgridGroundedFraction(), velocity_solver=solver)
    bed = -100.0 - 600.0 * X / 512e3 + 50.0 * _smooth((ny, nx), seed + 1, cells)
    H = 2000.0 * torch.sqrt(torch.clamp(1.0 - (X / 420e3) ** 2, min=0.0))
    Cf = 10.0 ** (6.5 + 0.3 * _smooth((ny, nx), seed + 2, cells)) * YEAR ** (1.0 / 3.0)
    return workloads.Case("sheet", grid, cfg, {}), dict(H=H.contiguous(), bed=bed, C=Cf, A=torch.full_like(H, 3.17e-24))


def _linear_inputs(case, seed):
    """The MISMIP+-like stream of the scaling benchmark at dx = 640 km / nx, its friction varied, and a stream's velocities."""
    ctl = dict(linear_iteration_control=nk.Convergence(reltol=1e-12, maxiter=50_000))
    c = workloads.mismip_stream(640e3 / case["nx"], velocity_solver=_solver(case, **ctl))
    ny, nx = case["ny"], case["nx"]
    f = {k: _t(v) for k, v in c.fields.items()}
    f["C"] = f["C"] * 10.0 ** (0.2 * _smooth((ny, nx), seed, nx / 32))
    x, y = _t(c.grid.faces(0))[None, :], _t(c.grid.centers(1))[:, None]
    u = 800.0 / YEAR * (x / 640e3) ** 2 * torch.exp(-((y - 40e3) / 24e3) ** 2)
    u = u * (1 + 0.1 * _smooth((ny, nx + 1), seed + 1, nx / 32))
    v = 20.0 / YEAR * _smooth((ny + 1, nx), seed + 2, nx / 32)
    u[:, 0] = 0
    u[:, -1] = 0
    v[0] = 0
    v[-1] = 0
    return c, f, u.contiguous(), v.contiguous()


def _transport_inputs(case, seed):
    """A sheet with a grounding line and an ice-free margin, and the velocities that carry it (at most a fifth of a cell
    a step)."""
    nx, ny = case["nx"], case["ny"]
    dx = 1000.0
    x = (torch.arange(nx, device=DEV, dtype=torch.float64)[None, :] + 0.5) / nx
    y = (torch.arange(ny, device=DEV, dtype=torch.float64)[:, None] + 0.5) / ny
    H = 1500.0 * torch.sqrt(torch.clamp(1 - (x / 0.9) ** 2, min=0.0)) * (1 + 0.1 * torch.cos(2 * math.pi * y))
    H = (H * (1 + 0.03 * _smooth((ny, nx), seed, 6.0))).clamp(min=0.0)
    bed = -200.0 - 900.0 * x + 60.0 * _smooth((ny, nx), seed + 1, 8.0)
    u = torch.zeros(ny, nx + 1, device=DEV, dtype=torch.float64)
    v = torch.zeros(ny + 1, nx, device=DEV, dtype=torch.float64)
    scale = 1000.0 / YEAR
    u[:, 1:-1] = scale * (0.3 + x[:, 1:] + 0.2 * _smooth((ny, nx - 1), seed + 2, 8.0))
    v[1:-1] = 0.3 * scale * _smooth((ny - 1, nx), seed + 3, 8.0)
    smb = 0.3 / YEAR * (1 + 0.5 * _smooth((ny, nx), seed + 4, 8.0))
    melt = 5.0 / YEAR * (1 + 0.5 * _smooth((ny, nx), seed + 5, 8.0)).clamp(min=0.0)
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * dx), y=(0.0, ny * dx), halo=(4, 4))
    cfg = dict(Nsigma=10, rheology=nk.GlenFlowLaw(rate_factor=3.17e-24), friction=nk.WeertmanFriction(),
               grounding=nk.SubgridGroundedFraction(), velocity_solver=nk.StressBalanceSolver())
    return grid, cfg, dict(H=H.contiguous(), bed=bed.contiguous(), u=u, v=v, smb=smb.contiguous(), melt=melt.contiguous()), 0.1 * YEAR


def _scheme(case):
    s = case.get("scheme", "weno")
    return {"weno": nk.WENO(order=5, bounds=(0.0, 1e5)), "weno unbounded": nk.WENO(order=5),
            "upwind 1": nk.UpwindBiased(order=1), "upwind 3": nk.UpwindBiased(order=3)}[s]


def _energy_inputs(case, seed):
    """A DIVA sheet's columns: cold to temperate ice, sheared velocities, a warm bed in part."""
    nx, ny, Ns = case["nx"], case["ny"], case["layers"]
    dx = 2000.0
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * dx), y=(0.0, ny * dx), halo=(4, 4))
    cfg = dict(Nsigma=Ns, stress_balance=nk.DepthIntegrated(shear=nk.DIVAShear(), side_walls=nk.FreeSlipWalls()),
               rheology=nk.GlenFlowLaw(rate_factor="sigma"), friction=nk.RegularizedCoulombFriction(),
               grounding=nk.SubgridGroundedFraction(), velocity_solver=nk.StressBalanceSolver())
    x = (torch.arange(nx, device=DEV, dtype=torch.float64)[None, :] + 0.5) / nx
    sm = lambda shape, k: _smooth(shape, seed + k, 8.0)  # noqa: E731
    H = (2000.0 * torch.sqrt(torch.clamp(1 - (x / 0.95) ** 2, min=0.0)) * (1 + 0.05 * sm((ny, nx), 0))).clamp(min=0.0)
    f = [(k / Ns) ** 2 for k in range(Ns + 1)]
    z = torch.tensor([(a + b) / 2 for a, b in zip(f, f[1:])], dtype=torch.float64, device=DEV)[:, None, None]
    T = 268.0 - 20.0 * z + 3.0 * sm((ny, nx), 1)
    Tpm = 273.15 - 7.9e-8 * 918.0 * 9.81 * H * (1 - z)
    E = 2009.0 * (torch.minimum(T, Tpm) - 223.15) + 3.34e5 * 0.005 * (sm((ny, nx), 2) > 1) * (z < 0.1)
    prof = 0.6 + 0.4 * (1 - (1 - z) ** 4)
    u = torch.zeros(ny, nx + 1, device=DEV, dtype=torch.float64)
    v = torch.zeros(ny + 1, nx, device=DEV, dtype=torch.float64)
    u[:, 1:-1] = 300.0 / YEAR * (0.2 + x[:, 1:] + 0.2 * sm((ny, nx - 1), 3))
    v[1:-1] = 50.0 / YEAR * sm((ny - 1, nx), 4)
    one = torch.ones(ny, nx, device=DEV, dtype=torch.float64)
    d = dict(H=H, u=u, v=v, u_b=0.6 * u, v_b=0.6 * v, u_sigma=prof * u, v_sigma=prof * v,
             beta_b_u=torch.where(u != 0, 3e9 * torch.exp(0.5 * sm((ny, nx + 1), 5)), torch.zeros_like(u)),
             beta_b_v=torch.where(v != 0, 3e9 * torch.exp(0.5 * sm((ny + 1, nx), 6)), torch.zeros_like(v)),
             eta_sigma=1e14 * (1 + z) * torch.exp(0.5 * sm((ny, nx), 7)), phi=((sm((ny, nx), 8) + 1.5) / 1.5).clamp(0.0, 1.0),
             T=torch.zeros(Ns, ny, nx, device=DEV, dtype=torch.float64), geothermal_flux=0.06 * (1 + 0.3 * sm((ny, nx), 9)),
             surface_temperature=250.0 + 5.0 * sm((ny, nx), 10), ocean_temperature=271.2 * one,
             basal_melt_rate=0.5 / YEAR * (1 + 0.5 * sm((ny, nx), 11)).clamp(min=0.0))
    state = dict(E=E.expand(Ns, ny, nx), Hw=0.05 * (1 + sm((ny, nx), 12)).clamp(min=0.0), H_previous=(H * (1 - 1e-3 * sm((ny, nx), 13))),
                 grounded_melt=1e-3 / YEAR * sm((ny, nx), 14).clamp(min=0.0))
    return grid, cfg, {k: a.contiguous() for k, a in d.items()}, {k: a.contiguous() for k, a in state.items()}, 0.5 * YEAR


# ---- prepare and run ------------------------------------------------------------------------------------------------
def _outputs(P, names):
    return {n: torch.empty(P.shape(n), dtype=torch.float64, device=DEV) for n in names}


def _set(P, fields):
    for n, a in fields.items():
        P.set_device(n, a.data_ptr())


def _get(P, out):
    """The fields of P into device arrays (nk_problem_get_field takes host or device memory)."""
    lib = library.load()
    for n, a in out.items():
        st = lib.nk_problem_get_field(P._h, abi.FIELD_IDS[n], C.cast(C.c_void_p(a.data_ptr()), C.POINTER(C.c_double)), a.numel())
        if st != abi.NK_OK:
            raise RuntimeError(f"nk_problem_get_field {n}: {abi.STATUS_NAMES[st]}")
    return out


def prepare(case, seed):
    seed = int(seed) * 7919 + 11
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("shelf", "sheet", "diva", "adjoint"):
        c, fields = _solve_inputs(case, seed)
        P = nk.Problem(c.grid, c.descriptors())
        s.update(P=P, zero={n: torch.zeros(P.shape(n), dtype=torch.float64, device=DEV) for n in ("u", "v")})
        if kind == "diva":   # the lagged state of the DIVA starts at rest too
            s["zero"].update({n: torch.zeros(P.shape(n), dtype=torch.float64, device=DEV) for n in ("beta_b_u", "beta_b_v", "F2", "eta_sigma")})
        s.update(fields=fields, out=_outputs(P, ("u", "v", "eta_H")))
        torch.cuda.synchronize()
        if kind == "adjoint":
            _set(P, fields)
            P.compute_geometry()
            P.picard_solve()
            u, v = P.get("u"), P.get("v")
            rng = np.random.default_rng(seed)
            ice = 1.0 + 0.1 * rng.standard_normal(u.shape)
            s["xbar"] = (u * ice * YEAR * YEAR, v * YEAR * YEAR)   # of half the squared misfit in (m/yr)^2
    elif kind == "linear":
        c, fields, u, v = _linear_inputs(case, seed)
        P = nk.Problem(c.grid, c.descriptors())
        torch.cuda.synchronize()
        _set(P, dict(fields, u=u, v=v))
        P.compute_geometry()
        P.update_coefficients()
        s.update(P=P, zero={n: torch.zeros(P.shape(n), dtype=torch.float64, device=DEV) for n in ("u", "v")},
                 b=(P.get("tau_u"), P.get("tau_v")), out=_outputs(P, ("u", "v")))
    elif kind in ("thickness", "gradient"):
        grid, cfg, f, dt = _transport_inputs(case, seed)
        P = nk.Problem(grid, nk.make_descriptors(grid, **cfg))
        torch.cuda.synchronize()
        _set(P, dict(H=f["H"], bed=f["bed"], u=f["u"], v=f["v"], surface_mass_balance=f["smb"], basal_melt_rate=f["melt"],
                     C=torch.full_like(f["H"], 1e9), A=torch.full_like(f["H"], 3.17e-24)))
        P.set_thickness_advection(_scheme(case))
        P.compute_geometry()
        s.update(P=P, dt=dt, start=dict(H=f["H"], u=f["u"], v=f["v"], clipped_thickness=torch.zeros_like(f["H"])),
                 out=_outputs(P, ("H", "clipped_thickness", "s", "phi", "tau_u", "tau_v")))
        torch.cuda.synchronize()
    elif kind == "energy":
        grid, cfg, f, state, dt = _energy_inputs(case, seed)
        P = nk.Problem(grid, nk.make_descriptors(grid, **cfg))
        torch.cuda.synchronize()
        _set(P, f)
        _set(P, state)
        s.update(P=P, dt=dt, start=state, out=_outputs(P, ("E", "T", "omega", "Hw", "grounded_melt", "basal_temperate_fraction",
                                                          "basal_heat_flux", "strain_heating")))
        torch.cuda.synchronize()
    else:
        sizes = [workloads.SERVING_SIZES[k % 4] for k in range(case["requests"])]
        s["cases"] = []
        for k, (nx, ny) in enumerate(sizes):
            c, f = _solve_inputs(dict(kind="sheet", nx=nx, ny=ny, precision="mixed", smoother="point"), seed + 31 * k)
            c.fields = {n: a.cpu().numpy() for n, a in f.items()}
            s["cases"].append(c)
        s["server"] = Server(max_in_flight=32, memory_cap_bytes=6 << 30)
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind in ("shelf", "sheet", "diva"):   # a request: its fields in, the geometry, the solve from rest, the velocities out
        P = s["P"]
        _set(P, s["fields"])
        if kind == "diva":
            P.compute_rate_factor()
        P.compute_geometry()
        _set(P, s["zero"])
        P.picard_solve()
        return _get(P, s["out"])
    if kind == "linear":
        P = s["P"]
        _set(P, s["zero"])
        P.linear_solve(*s["b"])
        return _get(P, s["out"])
    if kind == "adjoint":
        lu, lv, gc, ga, gh, _ = s["P"].picard_adjoint(*s["xbar"], thickness=True)
        return dict(lambda_u=lu, lambda_v=lv, log_C=gc, log_A=ga, H=gh)
    if kind == "thickness":
        P = s["P"]
        _set(P, s["start"])
        P.step_thickness(s["dt"])
        return _get(P, s["out"])
    if kind == "gradient":
        P, steps = s["P"], s["case"]["steps"]
        _set(P, s["start"])
        P.compute_geometry()
        g = P.checkpointed_gradient(lambda step, H, u, v, mask: (0.5 * float(np.sum(H * H)), H, None, None) if step == steps else None,
                                    s["dt"], steps, velocity_solves=False)
        return {n: g[n] for n in ("J", "H", "u", "v", "smb", "melt")}
    if kind == "energy":
        P = s["P"]
        _set(P, s["start"])
        P.step_enthalpy(s["dt"])
        return _get(P, s["out"])
    tickets = [s["server"].submit(c) for c in s["cases"]]
    return [s["server"].wait(t)[:2] for t in tickets]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def work(case):
    """bytes: every input field read once and every output written once.  flops: of the iterations that the stopping
    rules ask for (typical counts of these inputs), 42 a cell for the operator and 22 for the vectors of a CG step, 600
    for a V-cycle of two sweeps down and two up, 120 for a coefficient update."""
    kind = case["kind"]
    if kind == "serving":
        w = [work(dict(kind="sheet", nx=nx, ny=ny, precision="mixed", smoother="point"))
             for nx, ny in (workloads.SERVING_SIZES[k % 4] for k in range(case["requests"]))]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    n = case["nx"] * case["ny"]
    if kind == "shelf":
        return {"bytes": 8.0 * n * 8, "flops": float(n) * 40 * (120 + 250 * 64)}
    if kind == "sheet":
        return {"bytes": 9.0 * n * 8, "flops": float(n) * 40 * (120 + 20 * 664)}
    if kind == "diva":
        return {"bytes": (2 * 10 + 12.0) * n * 8, "flops": float(n) * 60 * (800 + 35 * 664)}
    if kind == "adjoint":
        return {"bytes": 14.0 * n * 8, "flops": float(n) * 50 * (400 + 30 * 664)}
    if kind == "linear":
        its = 1.2 * case["nx"] if case["preconditioner"] == "jacobi" else 40
        return {"bytes": 10.0 * n * 8, "flops": n * its * (64 if case["preconditioner"] == "jacobi" else 664)}
    if kind == "thickness":   # three stages: two reconstructions of about 60 operations at two faces of a cell
        return {"bytes": 13.0 * n * 8, "flops": 3.0 * n * (340 if case["scheme"].startswith("weno") else 120)}
    if kind == "gradient":
        return {"bytes": 12.0 * n * 8, "flops": case["steps"] * 3.0 * n * (2 * 340 + 1500)}
    Ns = case["layers"]
    return {"bytes": (8.0 * Ns + 14) * n * 8, "flops": float(n) * Ns * 90}


# ---- the same in plain 64-bit torch -----------------------------------------------------------------------------------
def _pad(a, x=0, y=0):
    """Edge values repeated x columns and y rows beyond the array (the zero-gradient halo)."""
    return torch.nn.functional.pad(a[None, None], (x, x, y, y), mode="replicate")[0, 0]


def _geometry(H, bed, rho_i=918.0, rho_w=1028.0, g=9.81):
    """Surface, effective pressure, ice mask, grounded fractions of centres and faces."""
    f = H + rho_w / rho_i * bed
    s = torch.maximum(bed + H, (1 - rho_i / rho_w) * H)
    N = (rho_i * g * H + rho_w * g * bed.clamp(max=0)).clamp(min=0)
    t = (H - 1.0).clamp(0, 1)
    mu = t * t * (3 - 2 * t)

    def segment(a, b):
        S = a.abs() + b.abs()
        return torch.where(S == 0, torch.ones_like(S), (a.clamp(min=0) + b.clamp(min=0)) / torch.where(S == 0, torch.ones_like(S), S))

    p = _pad(f, 1, 1)
    c, w, e, so, n = p[1:-1, 1:-1], p[1:-1, :-2], p[1:-1, 2:], p[:-2, 1:-1], p[2:, 1:-1]
    sw, se, nw, ne = p[:-2, :-2], p[:-2, 2:], p[2:, :-2], p[2:, 2:]

    def triangle(f1, f2, f3):
        a, hi = torch.minimum(torch.minimum(f1, f2), f3), torch.maximum(torch.maximum(f1, f2), f3)
        b = f1 + f2 + f3 - a - hi
        nz = lambda q: torch.where(q == 0, torch.ones_like(q), q)  # noqa: E731
        grounded = hi * hi / nz((hi - a) * (hi - b))
        floating = 1 - a * a / nz((b - a) * (hi - a))
        phi = torch.where(b > 0, floating, grounded)
        return torch.where(a >= 0, torch.ones_like(a), torch.where(hi <= 0, torch.zeros_like(a), phi))

    fe, fw, fn, fs = (c + e) / 2, (c + w) / 2, (c + n) / 2, (c + so) / 2
    fne, fnw, fse, fsw = (c + e + n + ne) / 4, (c + w + n + nw) / 4, (c + e + so + se) / 4, (c + w + so + sw) / 4
    phi = sum(triangle(c, a, b) for a, b in ((fe, fne), (fn, fne), (fn, fnw), (fw, fnw), (fw, fsw), (fs, fsw), (fs, fse), (fe, fse))) / 8
    px, py = _pad(f, x=1), _pad(f, y=1)
    return s, N, mu, phi, segment(px[:, :-1], px[:, 1:]), segment(py[:-1], py[1:])


def _driving_stress(H, s, mu, dx, dy, rho_i=918.0, rho_w=1028.0, g=9.81):
    D = (H - s).clamp(min=0).minimum(H)
    F = g * (rho_i * H * H - rho_w * D * D) / 2

    def component(H, s, mu, F, length, spacing):   # along the last axis, interior faces only
        a, b = mu[:, :-1], mu[:, 1:]
        west, east = (a > 0) & ~(b > 0), ~(a > 0) & (b > 0)
        front = length * (torch.where(west, F[:, :-1], 0 * a) - torch.where(east, F[:, 1:], 0 * a))
        t = -length * spacing * rho_i * g * (H[:, :-1] + H[:, 1:]) / 2 * (s[:, 1:] - s[:, :-1]) / spacing
        t = torch.where(west | east, front, t)
        return torch.nn.functional.pad(torch.where(a + b == 0, 0 * t, t), (1, 1))

    return component(H, s, mu, F, dy, dx), component(H.T, s.T, mu.T, F.T, dx, dy).T.contiguous()


class _Balance:
    """The SSA operator and its coefficients on a Bounded regular grid."""

    def __init__(self, case, fields, Lx, Ly, friction, eps0, wall_factor):
        self.ny, self.nx = fields["H"].shape
        self.dx, self.dy = Lx / self.nx, Ly / self.ny
        self.f, self.friction, self.eps0, self.wf = fields, friction, eps0, wall_factor
        self.s, self.N, self.mu, self.phi, self.phi_u, self.phi_v = _geometry(fields["H"], fields["bed"])
        self.tau = _driving_stress(fields["H"], self.s, self.mu, self.dx, self.dy)
        w = torch.ones(self.ny + 1, self.nx + 1, dtype=torch.float64, device=fields["H"].device)
        w[0], w[-1], w[:, 0], w[:, -1] = wall_factor, wall_factor, wall_factor, wall_factor
        self.corner = w

    def _shear(self, u, v):
        up, vp = torch.nn.functional.pad(u, (0, 0, 1, 1)), torch.nn.functional.pad(v, (1, 1))
        return self.corner * ((up[1:] - up[:-1]) / self.dy + (vp[:, 1:] - vp[:, :-1]) / self.dx) / 2

    def coefficients(self, u, v):
        H, dx, dy = self.f["H"], self.dx, self.dy
        un, vn = u.clone(), v.clone()
        un[:, 0], un[:, -1], vn[0], vn[-1] = 0, 0, 0, 0
        exx, eyy = (un[:, 1:] - un[:, :-1]) / dx, (vn[1:] - vn[:-1]) / dy
        e = self._shear(un, vn) ** 2
        ee = exx * exx + eyy * eyy + exx * eyy + (e[:-1, :-1] + e[:-1, 1:] + e[1:, :-1] + e[1:, 1:]) / 4 + self.eps0 ** 2
        self.eta = 0.5 * self.f["A"] ** (-1 / 3) * ee ** (-1 / 3) * H * self.mu
        p = _pad(self.eta, 1, 1)
        self.eta_ff = (p[:-1, :-1] + p[:-1, 1:] + p[1:, :-1] + p[1:, 1:]) / 4
        px, py = _pad(self.eta, x=1), _pad(self.eta, y=1)
        self.u_off, self.v_off = (px[:, :-1] + px[:, 1:]) == 0, (py[:-1] + py[1:]) == 0
        self.u_off[:, 0], self.u_off[:, -1], self.v_off[0], self.v_off[-1] = True, True, True, True
        if self.friction is None:
            self.bu, self.bv = torch.zeros_like(u), torch.zeros_like(v)
        else:
            vp, up = _pad(v, x=1), _pad(u, y=1)
            vf = (vp[:-1, :-1] + vp[:-1, 1:] + vp[1:, :-1] + vp[1:, 1:]) / 4
            uf = (up[:-1, :-1] + up[:-1, 1:] + up[1:, :-1] + up[1:, 1:]) / 4
            kind, m, u0, alpha2 = self.friction

            def drag(U, cell, mean):
                Cf = mean(self.f["C"])
                w = Cf * U ** (m - 1)
                if kind == "weertman":
                    return w
                tc = alpha2 * mean(self.N)
                return w * tc / (Cf ** (1 / m) * U + tc ** (1 / m)) ** m

            mx = lambda a: (_pad(a, x=1)[:, :-1] + _pad(a, x=1)[:, 1:]) / 2  # noqa: E731
            my = lambda a: (_pad(a, y=1)[:-1] + _pad(a, y=1)[1:]) / 2  # noqa: E731
            self.bu = self.phi_u * drag(torch.sqrt(u * u + vf * vf + u0 * u0), u, mx)
            self.bv = self.phi_v * drag(torch.sqrt(v * v + uf * uf + u0 * u0), v, my)
            self.bu[:, 0], self.bu[:, -1], self.bv[0], self.bv[-1] = 0, 0, 0, 0
        self.Az = dx * dy
        pu, pv = _pad(self.eta, x=1), _pad(self.eta, y=1)
        t = self.corner * self.eta_ff
        du = self.Az * self.bu + 4 * dy / dx * (pu[:, :-1] + pu[:, 1:]) + dx / dy * (t[:-1] + t[1:])
        dv = self.Az * self.bv + 4 * dx / dy * (pv[:-1] + pv[1:]) + dy / dx * (t[:, :-1] + t[:, 1:])
        self.du = torch.where(self.u_off | (du == 0), torch.ones_like(du), du)
        self.dv = torch.where(self.v_off | (dv == 0), torch.ones_like(dv), dv)
        self.u_on, self.v_on = (~self.u_off).to(u.dtype), (~self.v_off).to(v.dtype)

    def apply(self, u, v):
        dx, dy = self.dx, self.dy
        um, vm = u * self.u_on, v * self.v_on
        exx, eyy = (um[:, 1:] - um[:, :-1]) / dx, (vm[1:] - vm[:-1]) / dy
        sx, sy = 2 * dy * self.eta * (2 * exx + eyy), 2 * dx * self.eta * (2 * eyy + exx)
        t = 2 * self.eta_ff * self._shear(um, vm)
        sx, sy = torch.nn.functional.pad(sx, (1, 1)), torch.nn.functional.pad(sy, (0, 0, 1, 1))
        qu = self.Az * self.bu * u - (sx[:, 1:] - sx[:, :-1]) - dx * (t[1:] - t[:-1])
        qv = self.Az * self.bv * v - (sy[1:] - sy[:-1]) - dy * (t[:, 1:] - t[:, :-1])
        return torch.where(self.u_off, u, qu), torch.where(self.v_off, v, qv)

    def solve(self, u, v, reltol, maxiter):
        """Jacobi CG on A x = tau from (u, v), the residual tested every 20 steps."""
        bu, bv = self.tau
        au, av = self.apply(u, v)
        ru, rv = bu - au, bv - av
        zu, zv = ru / self.du, rv / self.dv
        pu, pv = zu, zv
        rho = (ru * zu).sum() + (rv * zv).sum()
        tol = reltol ** 2 * ((ru * ru).sum() + (rv * rv).sum())
        for k in range(maxiter):
            qu, qv = self.apply(pu, pv)
            alpha = rho / ((pu * qu).sum() + (pv * qv).sum())
            u, v = u + alpha * pu, v + alpha * pv
            ru, rv = ru - alpha * qu, rv - alpha * qv
            if k % 20 == 19 and bool((ru * ru).sum() + (rv * rv).sum() <= tol):
                break
            zu, zv = ru / self.du, rv / self.dv
            new = (ru * zu).sum() + (rv * zv).sum()
            pu, pv = zu + (new / rho) * pu, zv + (new / rho) * pv
            rho = new
        return u, v


def _weno(a, b, c, d, e):
    q0, q1, q2 = (2 * a - 7 * b + 11 * c) / 6, (-b + 5 * c + 2 * d) / 6, (2 * c + 5 * d - e) / 6
    b0 = 13 / 12 * (a - 2 * b + c) ** 2 + (a - 4 * b + 3 * c) ** 2 / 4
    b1 = 13 / 12 * (b - 2 * c + d) ** 2 + (b - d) ** 2 / 4
    b2 = 13 / 12 * (c - 2 * d + e) ** 2 + (3 * c - 4 * d + e) ** 2 / 4
    tau = (b0 - b2).abs()
    w = [g * (1 + tau / (bk + 1e-8)) for g, bk in ((0.1, b0), (0.6, b1), (0.3, b2))]
    return (w[0] * q0 + w[1] * q1 + w[2] * q2) / (w[0] + w[1] + w[2])


def _faces(H, scheme):
    """Reconstructions of H at the nx + 1 faces of every row, from the west and from the east cell."""
    n, p = H.shape[1], _pad(H, x=3)
    s = [p[:, k:k + n + 1] for k in range(6)]   # cells f - 3 .. f + 2 of face f
    if scheme.startswith("weno"):
        return _weno(*s[:5]), _weno(*s[:0:-1])
    if scheme == "upwind 3":
        return (-s[1] + 5 * s[2] + 2 * s[3]) / 6, (-s[4] + 5 * s[3] + 2 * s[2]) / 6
    return s[2], s[3]


def _thickness_stage(Hs, H0, u, v, smb, melt, bed, scheme, dtau, dx):
    phi = _geometry(Hs, bed)[3]
    xw, xe = _faces(Hs, scheme)
    ys, yn = (a.T for a in _faces(Hs.T, scheme))
    if scheme == "weno":   # the bounds-preserving limiter of every cell
        W, E, S, N = xe[:, :-1], xw[:, 1:], yn[:-1], ys[1:]
        w, eps = 5 / 18, 2 * 2.220446049250313e-16
        px, py = (Hs - w * W - w * E) / (1 - 2 * w), (Hs - w * S - w * N) / (1 - 2 * w)
        M = torch.maximum(torch.maximum(torch.maximum(px, py), torch.maximum(W, E)), torch.maximum(S, N))
        m = torch.minimum(torch.minimum(torch.minimum(px, py), torch.minimum(W, E)), torch.minimum(S, N))
        theta = torch.minimum(((1e5 - Hs) / (M - Hs + eps)).abs(), ((0.0 - Hs) / (m - Hs - eps)).abs()).clamp(max=1.0)
        hx, tx, hy, ty = _pad(Hs, x=1), _pad(theta, x=1), _pad(Hs, y=1), _pad(theta, y=1)
        xw, xe = hx[:, :-1] + tx[:, :-1] * (xw - hx[:, :-1]), hx[:, 1:] + tx[:, 1:] * (xe - hx[:, 1:])
        ys, yn = hy[:-1] + ty[:-1] * (ys - hy[:-1]), hy[1:] + ty[1:] * (yn - hy[1:])
    fx, fy = dx * u * torch.where(u > 0, xw, xe), dx * v * torch.where(v > 0, ys, yn)
    fx = torch.nn.functional.pad(fx[:, 1:-1], (1, 1))
    fy = torch.nn.functional.pad(fy[1:-1], (0, 0, 1, 1))
    div = (fx[:, 1:] - fx[:, :-1] + fy[1:] - fy[:-1]) / (dx * dx)
    star = H0 + dtau * (smb - (1 - phi) * melt - div)
    return star.clamp(min=0), (-star).clamp(min=0)


def _exact_transport(case, seed):
    _, _, f, dt = _transport_inputs(case, seed)
    scheme = case.get("scheme", "weno")
    names = ("H", "u", "v", "smb", "melt")
    H, u, v, smb, melt = inputs = [f[n].clone().requires_grad_(case["kind"] == "gradient") for n in names]

    def step(H):
        H0, clip = H, None
        for part in (1 / 3, 1 / 2, 1.0):
            H, clip = _thickness_stage(H, H0, u, v, smb, melt, f["bed"], scheme, part * dt, 1000.0)
        return H, clip

    if case["kind"] == "thickness":
        H, clip = step(H)
        s, _, mu, phi, _, _ = _geometry(H, f["bed"])
        tu, tv = _driving_stress(H, s, mu, 1000.0, 1000.0)
        return dict(H=H, clipped_thickness=clip, s=s, phi=phi, tau_u=tu, tau_v=tv)
    for _ in range(case["steps"]):
        H, _ = step(H)
    J = (H * H).sum() / 2
    return dict(zip(names, torch.autograd.grad(J, inputs)), J=float(J.detach()))


def _exact_energy(case, seed):
    _, _, f, st, dt = _energy_inputs(case, seed)
    Ns, dx, rho, g = case["layers"], 2000.0, 918.0, 9.81
    k_, c_, L, beta, T0, Tr, ratio, blend, wblend, Hmin, wmax, rate_max = (2.1, 2009.0, 3.34e5, 7.9e-8, 273.15, 223.15, 1e-3, 1.0, 1e-3,
                                                                           1.0, 0.01, 1.58443823077064e-9)
    zf = [(k / Ns) ** 2 for k in range(Ns + 1)]
    dz = [b - a for a, b in zip(zf, zf[1:])]
    zc = [(a + b) / 2 for a, b in zip(zf, zf[1:])]
    w2 = [((1 - a) ** 3 - (1 - b) ** 3) / 3 for a, b in zip(zf, zf[1:])]
    H, Hn, phi, E0, Hw, gm = f["H"], st["H_previous"], f["phi"], st["E"], st["Hw"], st["grounded_melt"]
    Epm = [c_ * (T0 - beta * rho * g * H * (1 - z) - Tr) for z in zc]
    ramp = lambda x, w: (x / w).clamp(0, 1)  # noqa: E731
    kap = []
    for k in range(Ns):
        w = ramp(E0[k] - Epm[k] + blend, blend)
        kap.append(k_ / c_ * (1 - w + w * ratio))
    u, v, ub, vb, bu, bv = f["u"], f["v"], f["u_b"], f["v_b"], f["beta_b_u"], f["beta_b_v"]
    exx, eyy = (u[:, 1:] - u[:, :-1]) / dx, (v[1:] - v[:-1]) / dx
    up, vp = torch.nn.functional.pad(u, (0, 0, 1, 1)), torch.nn.functional.pad(v, (1, 1))
    sh = ((up[1:] - up[:-1]) / dx + (vp[:, 1:] - vp[:, :-1]) / dx) / 2
    sh[0], sh[-1], sh[:, 0], sh[:, -1] = 0, 0, 0, 0   # free-slip walls
    sh = sh * sh
    e2 = exx * exx + eyy * eyy + exx * eyy + (sh[:-1, :-1] + sh[:-1, 1:] + sh[1:, :-1] + sh[1:, 1:]) / 4
    tb2 = (((bu * ub) ** 2)[:, :-1] + ((bu * ub) ** 2)[:, 1:]) / 2 + (((bv * vb) ** 2)[:-1] + ((bv * vb) ** 2)[1:]) / 2
    Phi = torch.stack([4 * f["eta_sigma"][k] * e2 + tb2 * w2[k] / (dz[k] * f["eta_sigma"][k]) for k in range(Ns)])
    Ht, Hnt = H.clamp(min=Hmin), Hn.clamp(min=Hmin)

    def div(q, k):   # of the upwind fluxes of q through layer k
        us, vs, qx, qy = f["u_sigma"][k], f["v_sigma"][k], _pad(q, x=1), _pad(q, y=1)
        fx, fy = dx * us * torch.where(us > 0, qx[:, :-1], qx[:, 1:]), dx * vs * torch.where(vs > 0, qy[:-1], qy[1:])
        fx, fy = torch.nn.functional.pad(fx[:, 1:-1], (1, 1)), torch.nn.functional.pad(fy[1:-1], (0, 0, 1, 1))
        return (fx[:, 1:] - fx[:, :-1] + fy[1:] - fy[:-1]) / (dx * dx)

    W = [-(1 - phi) * f["basal_melt_rate"] - gm]
    for k in range(Ns):
        W.append(W[-1] - dz[k] * ((Ht - Hnt) / dt + div(Hn, k)))
    D = kap[0] / (Ht * zc[0])
    F = ((bu * ub * ub)[:, :-1] + (bu * ub * ub)[:, 1:] + (bv * vb * vb)[:-1] + (bv * vb * vb)[1:]) / 2
    Epm_b, G = c_ * (T0 - beta * rho * g * H - Tr), f["geothermal_flux"]
    r = torch.maximum(ramp(E0[0] + (G + F) / D - Epm_b, blend), ramp(Hw, wblend))
    sb = ramp(E0[0] - Epm[0] + blend, blend)
    qg = phi * G + F
    mu = H > Hmin
    Es = c_ * (torch.minimum(f["surface_temperature"], torch.full_like(H, T0)) - Tr)
    Eo = c_ * (torch.minimum(f["ocean_temperature"], T0 - beta * rho * g * H) - Tr)
    chi, Fb = phi * r * (1 - sb), rho * W[0]
    Lam = D * (chi + 1 - phi) + (-Fb).clamp(min=0)
    S = (1 - r) * qg + D * (chi * Epm_b + (1 - phi) * Eo) + Fb.clamp(min=0) * Epm_b
    Fs, Ks = rho * W[Ns], kap[-1] / (Ht * (1 - zc[-1]))
    Ds, Ss = Ks + Fs.clamp(min=0), (Ks + (-Fs).clamp(min=0)) * Es
    low, upp = [], []   # the couplings of the interior faces
    for k in range(1, Ns):
        th = (zf[k] - zc[k - 1]) / (zc[k] - zc[k - 1])
        Fk = rho * W[k]
        cond = 1 / (Ht * ((zf[k] - zc[k - 1]) / kap[k - 1] + (zc[k] - zf[k]) / kap[k]))
        Dk = torch.maximum(cond, torch.maximum(Fk.clamp(min=0) * th, (-Fk).clamp(min=0) * (1 - th)))
        low.append(-Fk * (1 - th) - Dk)
        upp.append(Fk * th - Dk)
    zero, one = torch.zeros_like(H), torch.ones_like(H)
    cp, dp = [], []
    for k in range(Ns):
        dm = Lam if k == 0 else -upp[k - 1]
        dq = Ds if k == Ns - 1 else -low[k]
        force = (S if k == 0 else zero) + (Ss if k == Ns - 1 else zero)
        b = torch.where(mu, rho * Ht * dz[k] / dt + dm + dq, one)
        transport = zero
        us, vs = f["u_sigma"][k], f["v_sigma"][k]
        hx, hy, qx, qy = _pad(Hn, x=1), _pad(Hn, y=1), _pad(E0[k], x=1), _pad(E0[k], y=1)
        fx = dx * us * torch.where(us > 0, hx[:, :-1] * qx[:, :-1], hx[:, 1:] * qx[:, 1:])
        fy = dx * vs * torch.where(vs > 0, hy[:-1] * qy[:-1], hy[1:] * qy[1:])
        transport = rho * dz[k] * (fx[:, 1:] - fx[:, :-1] + fy[1:] - fy[:-1]) / (dx * dx)
        rhs = torch.where(mu, rho * Hnt * dz[k] * E0[k] / dt - transport + Ht * dz[k] * Phi[k] + force, Es)
        # row k + 1 couples down through low[k], row k up through upp[k]
        up_k = torch.where(mu, upp[k], zero) if k < Ns - 1 else zero
        if k == 0:
            piv = b
            dp.append(rhs / piv)
        else:
            lo_k = torch.where(mu, low[k - 1], zero)
            piv = b - lo_k * cp[-1]
            dp.append((rhs - lo_k * dp[-1]) / piv)
        cp.append(up_k / piv)
    e = [None] * Ns
    e[-1] = dp[-1]
    for k in range(Ns - 2, -1, -1):
        e[k] = dp[k] - cp[k] * e[k + 1]
    melt = r * (qg - phi * (1 - sb) * D * (Epm_b - e[0])) / (rho * L)
    drained = zero
    for k in range(Ns):
        w = (e[k] - Epm[k]).clamp(min=0) / L
        rate = rate_max * ((w / wmax - 1).clamp(0, 1) + 9 * (w / wmax - 2).clamp(0, 1)) / 10
        dw = torch.where(mu, torch.minimum(dt * rate, (w - wmax).clamp(min=0)), zero)
        e[k] = e[k] - L * dw
        drained = drained + Ht * dz[k] * dw
    star = Hw + dt * torch.where(mu, melt, zero) + drained
    plus = star.clamp(min=0)
    e[0] = e[0] - L * (plus - star) / (Ht * dz[0])
    E = torch.stack(e)
    T = torch.stack([torch.minimum(T0 - beta * rho * g * H * (1 - zc[k]), Tr + e[k] / c_) for k in range(Ns)])
    om = torch.stack([(e[k] - Epm[k]).clamp(min=0) / L for k in range(Ns)])
    return dict(E=E, T=T, omega=om, Hw=plus, grounded_melt=(plus - Hw) / dt, basal_temperate_fraction=sb, basal_heat_flux=qg, strain_heating=Phi)


def exact(case, seed):
    seed = int(seed) * 7919 + 11
    kind = case["kind"]
    if kind in ("thickness", "gradient"):
        return _exact_transport(case, seed)
    if kind == "energy":
        return _exact_energy(case, seed)
    if kind == "linear":
        _, f, u, v = _linear_inputs(case, seed)
        B = _Balance(case, f, 640e3, 80e3, ("coulomb", 1.0 / 3.0, 1e-5 / YEAR, 0.5), 1e-5 / YEAR, 0.0)
        B.coefficients(u, v)
        u, v = B.solve(torch.zeros_like(u), torch.zeros_like(v), 1e-13, 20_000)
        return dict(u=u, v=v)
    if kind in ("shelf", "sheet") and case["nx"] * case["ny"] <= 9000:   # larger ones take too long this way
        c, f = _solve_inputs(case, seed)
        drag = None if kind == "shelf" else ("weertman", 1.0 / 3.0, 1e-8, 0.0)
        B = _Balance(case, f, c.grid.x[1], c.grid.y[1], drag, 1e-13, 2.0 if kind == "shelf" else 0.0)
        u, v = torch.zeros(B.ny, B.nx + 1, dtype=torch.float64, device=DEV), torch.zeros(B.ny + 1, B.nx, dtype=torch.float64, device=DEV)
        for _ in range(100):
            B.coefficients(u, v)
            a, b = B.solve(u, v, 1e-8, 10_000)
            change, norm = torch.sqrt(((a - u) ** 2).sum() + ((b - v) ** 2).sum()), torch.sqrt((a * a).sum() + (b * b).sum())
            u, v = a, b
            if bool(change <= 1e-6 * norm):
                break
        return dict(u=u, v=v, eta_H=B.eta)
    return None
