"""One-step IMEX and the adaptive chemistry on both sides of the temperatures
between which the specialised rates' straight-line quotients hold (150 K and
1e4 K: outside, the cell takes the table-driven form), in one launch whose
warps mix both, against the oracle; 33 x 5 x 3 cells leave partial warps.

Tolerance: the repository's bar for one call, 1e-12 of each variable's largest
magnitude (the two forms differ by the order of a few roundings)."""
import numpy as np
import pytest

from _cases import QUIRKS_FIXED, interior, make_oracle, rel_err
from eu3d_b200 import gpu
from eu3d_b200.readers import make_grid

pytestmark = pytest.mark.gpu
TOL_FN = 1e-12


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("window", [(120.0, 190.0), (9700.0, 10300.0), (149.9, 150.1)], ids=["cold", "hot", "edge"])
def test_imex_outside_the_fast_range(mech, window, bits):
    g = make_grid(33, 0.0, 0.01, 5, 0.0, 0.006, 3, 0.0, 0.004, 2, fixed_ghosts=True)
    o, g = make_oracle(mech, seed=6, quirks=QUIRKS_FIXED, grid=g, tlo=window[0], thi=window[1], radicals=1e-6)
    d = gpu.DeviceFlowfield(mech, g, quirks=QUIRKS_FIXED, flux_bits=bits)
    d.upload_state(o)
    o.update_after_cs()
    d.update_after_cs()
    T = interior(o.view("T"))
    assert (T < 150.0).any() or (T > 1e4).any()
    o.partial_t()
    o.dt = 1e-12
    d.dt = 1e-12
    o.imex()
    d.imex()
    for n in ("CS", "T"):
        e = rel_err(interior(d.download(n)), interior(o.view(n)))
        assert e < TOL_FN, (n, e)
    assert d.status()["nonfinite_cells"] == 0
