"""Ghost fills of grids with extents of one and two cells.  With one cell along
an axis the mirror image of an outer ghost cell is a ghost cell of the other
end, so the result depends on the order of the fill: the reference's, x, y, z,
each from the lowest index up.  Every ghost cell of every field against the
oracle, after two fills (the second takes what the first left).

Tolerances: FP64 the repository's bar for one call (1e-12 of each variable's
largest magnitude); FP32 primitives 1e-6: inputs rounded to 6e-8 each, through
D = P / (T R), and sums over nine species whose terms stay within ten times
the sum."""
import numpy as np
import pytest

import golden.make_golden as mg
from _cases import QUIRKS_FIXED, make_oracle, rel_err
from eu3d_b200 import gpu
from eu3d_b200.readers import make_grid

pytestmark = pytest.mark.gpu

EXTENTS = [(1, 1, 1), (1, 5, 4), (6, 1, 4), (6, 5, 1), (2, 1, 33), (1, 2, 1), (2, 2, 2)]


def grid(ni, nj, nk):
    g = make_grid(max(ni, 2), 0.0, 0.01, max(nj, 2), 0.0, 0.006, max(nk, 2), 0.0, 0.004, 2, fixed_ghosts=True)
    g.ni, g.nj, g.nk = ni, nj, nk
    g.xnode, g.ynode, g.znode = g.xnode[:ni + 4].copy(), g.ynode[:nj + 4].copy(), g.znode[:nk + 4].copy()
    return g


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("kind", [gpu.BC_RSBI, gpu.BC_ODM, gpu.BC_TRANSMISSIVE], ids=["rsbi", "odm", "transmissive"])
@pytest.mark.parametrize("dims", EXTENTS, ids=lambda d: "x".join(map(str, d)))
def test_ghosts_of_thin_grids(mech, dims, kind, bits):
    o, g = make_oracle(mech, seed=21, quirks=QUIRKS_FIXED, grid=grid(*dims), tlo=1100.0, thi=2600.0)
    d = gpu.DeviceFlowfield(mech, g, quirks=QUIRKS_FIXED, flux_bits=bits)
    d.upload_state(o)
    if kind == gpu.BC_ODM:
        mg.set_inflow(o)
        d.set_inflow(*[o.view(n) for n in ("Uint", "Vint", "Wint", "Pint", "Dint", "Tint", "Hint", "Eint", "Gint",
                                           "Yint")])
    for _ in range(2):
        o.boundary(kind)
        d.boundary(kind)
        for n in ("U", "V", "W", "P", "D", "T", "H", "Gamma", "E", "Yi"):
            assert rel_err(d.download(n), o.view(n)) < (1e-12 if bits == 64 else 1e-6), n
    d.close()
