"""A NaN in one passive field reaches the residuals it reaches in the oracle,
whatever its sign and the flow's direction.  The passive fields (tangential
velocities, H, species) are reconstructed on the upwind side alone and enter
neither the pressure nor the mass flux, so that only the limiter can spread or
drop it: a NaN in the cell downwind of a face must reach the upwind state
through the slope.  The last case makes the slope's divisor zero (a difference
of exactly -1e-12), which is a NaN in the reference's formula too."""
import numpy as np
import pytest

from _cases import QUIRKS_FIXED, interior, make_oracle
from eu3d_b200 import gpu
from eu3d_b200.readers import make_grid

pytestmark = pytest.mark.gpu

NEG_NAN = np.array([0xFFF8000000000000], dtype=np.uint64).view(np.float64)[0]
AT = (20, 6, 4)


@pytest.mark.parametrize("diff", [gpu.DIFF_MUSCL1, gpu.DIFF_MUSCL2, gpu.DIFF_WENO], ids=["muscl1", "muscl2", "weno"])
@pytest.mark.parametrize("flow", [1.0, -1.0], ids=["up", "down"])
@pytest.mark.parametrize("what", ["H+", "H-", "Y+", "Y-", "divisor"])
def test_nan_in_one_passive_field(mech, what, flow, diff):
    g = make_grid(37, 0.0, 0.01, 9, 0.0, 0.006, 5, 0.0, 0.004, 2, fixed_ghosts=True)
    o, g = make_oracle(mech, seed=4, quirks=QUIRKS_FIXED, grid=g, tlo=1100.0, thi=2600.0)
    for n in ("U", "V", "W"):
        o.view(n)[...] = flow * (50.0 + np.abs(o.view(n)))
    nan = NEG_NAN if what.endswith("-") else np.nan
    if what[0] == "H":
        o.view("H")[AT] = nan
    elif what[0] == "Y":
        o.view("Yi")[AT + (3,)] = nan
    else:
        # a face's divisor is (next - this) + 1e-12 on its left, where `this` is the far
        # cell, and the same with the far cell last on its right
        y = o.view("Yi")[..., 3]
        y[18:23, 6, 4] = [1e-12, 0.0, 0.25, 1e-12, 0.0]
    d = gpu.DeviceFlowfield(mech, g, quirks=QUIRKS_FIXED, flux_bits=64)
    d.upload_state(o)
    o.dt = d.dt = 1e-9
    o.advection(0, diff)
    d.advection(0, diff)
    a, b = interior(d.download("RHS")), interior(o.view("RHS"))
    if diff == gpu.DIFF_MUSCL2 or what != "divisor":
        assert np.isnan(b).any()
    assert not np.isnan(b).all(axis=(0, 1, 2)).any()
    assert np.array_equal(np.isnan(a), np.isnan(b))
    d.close()
