"""The FP64 flux's walk along z: flux_kz is a limit that a launch shortens on
small grids, so that every setting the autotuner can keep runs them as well as
the one a handle begins with; and walks of several planes, which take a grid
of some size, give the bits of single planes."""
import numpy as np
import pytest

from _cases import QUIRKS_FIXED, interior, make_oracle
from eu3d_b200 import gpu
from eu3d_b200.readers import make_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(241, 81, 2), (400, 2, 2), (24, 12, 20), (160, 60, 40)], ids=lambda d: "x".join(map(str, d)))
def test_a_handle_begins_with_a_setting_the_autotuner_tries(mech, dims):
    g = make_grid(dims[0], 0.0, 0.01, dims[1], 0.0, 0.006, dims[2], 0.0, 0.004, 2, fixed_ghosts=True)
    o, g = make_oracle(mech, seed=3, quirks=QUIRKS_FIXED, grid=g, tlo=1100.0, thi=1500.0)
    d = gpu.DeviceFlowfield(mech, g, quirks=QUIRKS_FIXED, flux_bits=64)
    d.upload_state(o)
    first = d.tuning()
    assert first["flux_kz"] in (4, 8, 16, 32, 64)
    # a setting outside the candidates competes too, and the best is one of these
    d.set_tuning(flux_kz=5)
    d.dt = 1e-9
    best, ms = d.autotune(steps=2, react=gpu.REACT_IMEX, bc_kind=gpu.BC_RSBI)
    assert best["flux_kz"] in (4, 5, 8, 16, 32, 64) and ms > 0
    d.close()


@pytest.mark.parametrize("diff", [gpu.DIFF_MUSCL2, gpu.DIFF_WENO], ids=["muscl2", "weno"])
def test_walks_of_several_planes_give_the_bits_of_one(mech, diff):
    # 3 x 100 tiles of 32 x 7 columns: walks of 1, 4 (two full, one of one plane) and 8 planes stay as they are set
    dims = (96, 700, 9)
    g = make_grid(dims[0], 0.0, 0.01, dims[1], 0.0, 0.06, dims[2], 0.0, 0.004, 2, fixed_ghosts=True)
    o, g = make_oracle(mech, seed=5, quirks=QUIRKS_FIXED, grid=g, tlo=1100.0, thi=2600.0)
    d = gpu.DeviceFlowfield(mech, g, quirks=QUIRKS_FIXED, flux_bits=64)
    d.upload_state(o)
    d.dt = 1e-9
    out = []
    for kz in (1, 4, 8):
        d.set_tuning(flux_kz=kz)
        d.advection(0, diff)
        out.append(interior(d.download("RHS")).copy())
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    d.close()
