"""The one-thread-per-cell kernels number their warps through over all rows, a
32-cell segment of an x row each: whole steps against the oracle at row lengths
around one, two and four segments, and rows shorter than a warp, with every
time scheme (the SSP stage updates) and both one-step chemistries.

Tolerance: the repository's bar for a few steps, 1e-10 of each variable's
largest magnitude."""
import numpy as np
import pytest

from _cases import QUIRKS_FIXED, interior, make_oracle
from eu3d_b200 import gpu
from eu3d_b200.readers import make_grid
from test_gpu_parity import TOL_STEP, to_gpu, worst

pytestmark = pytest.mark.gpu

ROWS = [(3, 5, 3), (31, 3, 2), (32, 3, 2), (33, 2, 3), (64, 2, 2), (65, 3, 2), (129, 2, 2)]


@pytest.mark.parametrize("adv", [gpu.ADV_EE, gpu.ADV_SSPRK2, gpu.ADV_SSPRK3], ids=["ee", "rk2", "rk3"])
@pytest.mark.parametrize("dims", ROWS, ids=lambda d: "x".join(map(str, d)))
def test_steps_at_ragged_row_lengths(mech, dims, adv):
    g = make_grid(dims[0], 0.0, 0.001 * dims[0], dims[1], 0.0, 0.001 * dims[1], dims[2], 0.0, 0.001 * dims[2], 2,
                  fixed_ghosts=True)
    o, g = make_oracle(mech, seed=16, quirks=QUIRKS_FIXED, grid=g, tlo=1100.0, thi=1500.0)
    d = to_gpu(o, g, QUIRKS_FIXED)
    for _ in range(3):
        o.step(gpu.REACT_IMEX, 0, adv, gpu.DIFF_MUSCL2, 0.3, 1.0, gpu.BC_RSBI)
        d.step(react=gpu.REACT_IMEX, timeadv=adv, diff=gpu.DIFF_MUSCL2, bc_kind=gpu.BC_RSBI, cfl=0.3)
    assert np.isfinite(interior(o.view("T"))).all()
    e, errs = worst(d, o)
    assert e < TOL_STEP, errs
    d.close()


@pytest.mark.parametrize("dims", [(31, 3, 2), (33, 2, 3), (65, 3, 2)], ids=lambda d: "x".join(map(str, d)))
def test_trapezoid_at_ragged_row_lengths(mech, dims):
    g = make_grid(dims[0], 0.0, 0.001 * dims[0], dims[1], 0.0, 0.001 * dims[1], dims[2], 0.0, 0.001 * dims[2], 2,
                  fixed_ghosts=True)
    o, g = make_oracle(mech, seed=17, quirks=QUIRKS_FIXED, grid=g, tlo=450.0, thi=530.0)
    d = to_gpu(o, g, QUIRKS_FIXED)
    for type_ in (0, 1):
        for x in (o, d):
            x.dt = 5e-9
            x.boundary(gpu.BC_RSBI)
            x.advection(0, gpu.DIFF_MUSCL2)
            x.trapezoid(type_)
    assert np.isfinite(interior(o.view("T"))).all()
    e, errs = worst(d, o)
    assert e < TOL_STEP, errs
    d.close()
