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
