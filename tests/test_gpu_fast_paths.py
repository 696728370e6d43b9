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
