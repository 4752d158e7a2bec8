"""The FP64 flux kernel's division-free reconstruction and AUSM against the
oracle's quotients, at the edges of its tiles (32 x 7 and 32 x 3 columns, walks
of kz planes): one advection, relative to each variable's largest residual.

Tolerance: the repository's bar for one call, 1e-12 of the largest magnitude
of each variable.  A face flux carries a few ulp (1e-15) of its own size, and
the noise of the state keeps the largest residual of every variable within two
orders of the flux differences it is formed from."""
import numpy as np
import pytest

from _cases import QUIRKS_FIXED, QUIRKS_REF, interior, make_oracle, rel_err
from eu3d_b200 import gpu
from eu3d_b200.readers import make_grid

pytestmark = pytest.mark.gpu
TOL_FN = 1e-12

SIZES = [((33, 8, 5), 1), ((32, 7, 4), 4), ((31, 6, 3), 2), ((65, 3, 2), 1), ((5, 2, 2), 16), ((1, 1, 1), 1),
         ((96, 29, 34), 1), ((95, 64, 20), 1)]


@pytest.mark.parametrize("diff", [gpu.DIFF_MUSCL1, gpu.DIFF_MUSCL2, gpu.DIFF_WENO], ids=["muscl1", "muscl2", "weno"])
@pytest.mark.parametrize("dims,kz", SIZES, ids=[f"{d[0]}x{d[1]}x{d[2]}-kz{k}" for d, k in SIZES])
def test_flux64_tiles(mech, dims, kz, diff):
    quirks = QUIRKS_REF if dims[0] == 33 else QUIRKS_FIXED
    g = make_grid(dims[0], 0.0, 0.01, dims[1], 0.0, 0.006, dims[2], 0.0, 0.004, 2, fixed_ghosts=True) \
        if min(dims) > 1 else _single_cell()
    hot = dict(tlo=1100.0, thi=2600.0) if quirks == QUIRKS_FIXED else dict(tlo=450.0, thi=980.0)
    o, g = make_oracle(mech, seed=sum(dims), quirks=quirks, grid=g, **hot)
    d = gpu.DeviceFlowfield(mech, g, quirks=quirks, flux_bits=64)
    d.upload_state(o)
    d.set_tuning(flux_kz=kz)
    o.dt = 1e-9
    d.dt = 1e-9
    o.advection(0, diff)
    d.advection(0, diff)
    e = rel_err(interior(d.download("RHS")), interior(o.view("RHS")))
    assert e < TOL_FN, e


def _single_cell():
    g = make_grid(2, 0.0, 0.001, 2, 0.0, 0.001, 2, 0.0, 0.001, 2, fixed_ghosts=True)
    x = np.arange(-2, 3) * 0.001
    g.ni = g.nj = g.nk = 1
    g.xnode = g.ynode = g.znode = x
    return g


def test_flux64_nan_spreads_as_in_the_oracle(mech):
    """A NaN in one cell's primitives reaches the same residuals."""
    g = make_grid(37, 0.0, 0.01, 9, 0.0, 0.006, 5, 0.0, 0.004, 2, fixed_ghosts=True)
    o, g = make_oracle(mech, seed=4, quirks=QUIRKS_FIXED, grid=g, tlo=1100.0, thi=2600.0)
    for n in ("P", "Gamma", "U", "H"):
        o.view(n)[20, 6, 4] = np.nan
    o.view("Yi")[20, 6, 4] = np.nan
    d = gpu.DeviceFlowfield(mech, g, quirks=QUIRKS_FIXED, flux_bits=64)
    d.upload_state(o)
    o.dt = d.dt = 1e-9
    o.advection(0, gpu.DIFF_MUSCL2)
    d.advection(0, gpu.DIFF_MUSCL2)
    a, b = interior(d.download("RHS")), interior(o.view("RHS"))
    assert np.isnan(b).any() and np.array_equal(np.isnan(a), np.isnan(b))
