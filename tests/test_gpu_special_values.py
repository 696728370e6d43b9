"""Infinities and NaN in fields that the FP64 kernels test on the integer units: the oracle's comparisons decide."""
import numpy as np
import pytest

import nunatak_gb300 as nk
from support import make

gpu = pytest.mark.gpu


# A face whose velocity is +inf is an eastward (northward) one, so its flux takes the thickness behind it: the cell behind
# empties and the one before it is filled without bound, also where it was empty.
@gpu
@pytest.mark.parametrize("component, value", [("u", np.inf), ("u", -np.inf), ("v", np.inf), ("v", -np.inf), ("u", np.nan)])
@pytest.mark.parametrize("scheme", [nk.UpwindBiased(order=1), nk.WENO(order=5)])
def test_an_unbounded_velocity_is_upwinded(oracle_cls, gpu_cls, component, value, scheme):
    nx, ny = 12, 9
    grid = nk.RectilinearGrid(size=(nx, ny), x=(0.0, nx * 1e3), y=(0.0, ny * 1e3), halo=(4, 4))
    H = np.full((ny, nx), 500.0)
    H[5:, :] = 0.0
    H[:, 7:] = 0.0
    out = []
    for cls in (gpu_cls, oracle_cls):
        P = make(cls, grid, advection=scheme, rheology=nk.GlenFlowLaw(rate_factor=3e-24), friction=nk.WeertmanFriction())
        w = np.zeros(P.shape(component))
        w[(2, 7) if component == "u" else (5, 2)] = value
        for n, a in (("H", H), ("bed", 10.0), (component, w)):
            P.set(n, a)
        P.compute_geometry()
        P.step_thickness_stage(1e5, 1)   # at rest elsewhere: whole numbers
        out.append(P.get("H"))
        P.close()
    assert np.array_equal(out[0], out[1], equal_nan=True)
    assert not value > 0 or np.any(np.isinf(out[1]))


# A column whose enthalpy is NaN holds no water: max(0, E - E_pm) keeps its first operand, in the diagnosed fraction as in
# what drains.  The other column, at rest beside it, is untouched.  (E, T and ω; 1e-10 as in the energy step's other tests.)
@gpu
def test_nan_enthalpy_holds_no_water(oracle_cls, gpu_cls):
    grid = nk.RectilinearGrid(size=(2, 1), x=(0.0, 2e3), y=(0.0, 1e3))
    out = []
    for cls in (gpu_cls, oracle_cls):
        P = make(cls, grid, Nsigma=6, rheology=nk.GlenFlowLaw(rate_factor="sigma"), friction=nk.WeertmanFriction())
        E = np.full((6, 1, 2), 2009.0 * 51.0)   # temperate
        E[3, 0, 0] = np.nan
        for n, a in (("H", 1000.0), ("bed", 10.0), ("E", E)):
            P.set(n, a)
        P.compute_geometry()
        for n, a in (("geothermal_flux", 0.042), ("surface_temperature", 243.15), ("ocean_temperature", 271.15), ("H_previous", 1000.0),
                     ("Hw", 0.0), ("basal_melt_rate", 0.0)):
            P.energy_set(n, a)
        P.step_enthalpy(1e7)
        out.append([P.get(n) for n in ("E", "T", "omega")] + [P.energy_get(n) for n in ("Hw", "grounded_melt")])
        P.close()
    for g, w in zip(*out):
        assert np.allclose(g, w, rtol=1e-10, atol=0.0, equal_nan=True)
    assert np.all(np.isnan(out[1][0][:, 0, 0])) and np.all(out[1][2][:, 0, 0] == 0.0) and np.any(out[1][2][:, 0, 1] > 0.0)
