"""Where the chemistry's straight-line quotients stop and IEEE division takes
over: the adaptive integrator on both sides of 90 K and 1e4 K (a cell outside
takes the table-driven rates and IEEE quotients, in one launch whose warps mix
both), one-step IMEX on both sides of 90 K and at densities below 1e-30, the
bits of cold cells within the range, and a mechanism other than the
compiled-in one, whose rates are unbounded: its implicit update divides by
denominators past the largest number and must give what the oracle gives, an
update of zero, and not a NaN.

Tolerances: one IMEX call 1e-12 of each variable's largest magnitude, the
repository's bar; an adaptive step 1e-8, its bar against the oracle (the two
sum in different orders, and a substep's length follows the state).  Cold
cells: golden/cold_chem.npz holds what an implementation with the compiler's
divisions recorded on a B200, whose bits the straight-line quotients give."""
import copy
import os

import numpy as np
import pytest

from adaptive_oracle import adaptive_step
from _cases import QUIRKS_FIXED, fill_state, interior, make_oracle, rel_err
from eu3d_b200 import gpu
from eu3d_b200 import surrogate as S
from eu3d_b200.readers import make_grid
from pyoracle import Oracle

pytestmark = pytest.mark.gpu
TOL_FN, TOL_ADAPT = 1e-12, 1e-8


# 33 cells a row leave a warp with one cell
def _grid():
    return make_grid(33, 0.0, 0.01, 5, 0.0, 0.006, 3, 0.0, 0.004, 2, fixed_ghosts=True)


LOW, HIGH = 90.0, 1e4
WINDOWS = {"cold": (80.0, 120.0, 1e-12), "hot": (9700.0, 10300.0, 1e-13), "edge": (89.9, 90.1, 1e-12)}
GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "cold_chem.npz")


@pytest.mark.parametrize("generic", [False, True], ids=["compiled-in", "table"])
@pytest.mark.parametrize("window", WINDOWS)
def test_adaptive_outside_the_fast_range(mech, window, generic, monkeypatch):
    if generic:
        monkeypatch.setenv("EU3D_GENERIC_CHEM", "1")
    lo, hi, dt = WINDOWS[window]
    o, g = make_oracle(mech, seed=6, quirks=QUIRKS_FIXED, grid=_grid(), tlo=lo, thi=hi, radicals=1e-6)
    d = gpu.DeviceFlowfield(mech, g, quirks=QUIRKS_FIXED, flux_bits=64)
    d.upload_state(o)
    o.update_after_cs()
    d.update_after_cs()
    T = interior(o.view("T"))
    assert ((T < LOW) | (T > HIGH)).any() and ((T > LOW) & (T < HIGH)).any()
    o.view("RHS")[...] = 0.0
    d.upload("RHS", np.zeros(d.shape("RHS")))
    d.set_elements(S.atoms_matrix(mech))
    o.dt = d.dt = dt
    n = adaptive_step(o, dt, S.atoms_matrix(mech))
    d.react_adaptive()
    for f in ("CS", "T"):
        e = rel_err(interior(d.download(f)), interior(o.view(f)))
        assert e < TOL_ADAPT, (f, e)
    st = d.status()
    assert st["nonfinite_cells"] == 0
    # a rounding may move a substep boundary of a cell
    assert abs(st["substeps"] - int(n.sum())) <= 0.01 * n.sum()
    d.close()


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("window", ["cold", "edge"])
def test_imex_around_the_lower_end(mech, window, bits):
    lo, hi, dt = WINDOWS[window]
    o, g = make_oracle(mech, seed=6, quirks=QUIRKS_FIXED, grid=_grid(), tlo=lo, thi=hi, radicals=1e-6)
    d = gpu.DeviceFlowfield(mech, g, quirks=QUIRKS_FIXED, flux_bits=bits)
    d.upload_state(o)
    o.update_after_cs()
    d.update_after_cs()
    T = interior(o.view("T"))
    assert (T < LOW).any() and (T > LOW).any()
    o.partial_t()
    o.dt = d.dt = dt
    o.imex()
    d.imex()
    for f in ("CS", "T"):
        e = rel_err(interior(d.download(f)), interior(o.view(f)))
        assert e < TOL_FN, (f, e)
    d.close()


def cold_chemistry(mech):
    """CS and T of cells between 92 and 170 K after one IMEX and one adaptive step."""
    out = {}
    for react in ("imex", "adaptive"):
        g = make_grid(33, 0.0, 0.01, 3, 0.0, 0.006, 2, 0.0, 0.004, 2, fixed_ghosts=True)
        o, g = make_oracle(mech, seed=8, quirks=QUIRKS_FIXED, grid=g, tlo=92.0, thi=170.0, radicals=1e-4)
        d = gpu.DeviceFlowfield(mech, g, quirks=QUIRKS_FIXED, flux_bits=64)
        d.upload_state(o)
        d.update_after_cs()
        d.upload("RHS", np.zeros(d.shape("RHS")))
        d.set_elements(S.atoms_matrix(mech))
        d.dt = 1e-8
        d.imex() if react == "imex" else d.react_adaptive()
        out[react] = np.concatenate([interior(d.download("CS")), interior(d.download("T"))[..., None]], axis=-1)
        d.close()
    return out


def test_cold_cells_keep_the_bits_of_plain_divisions(mech):
    got, want = cold_chemistry(mech), np.load(GOLDEN)
    for react, v in got.items():
        assert want[react][..., -1].min() > LOW and (want[react][..., -1] < 150.0).any()
        assert np.array_equal(v, want[react]), react


def test_queue_of_the_table_form_matches_thread_per_cell(mech, monkeypatch):
    """The persistent queue, compiled for other resident blocks with the table-driven
    rates, against one thread per cell: the same substeps, the state to rounding."""
    monkeypatch.setenv("EU3D_GENERIC_CHEM", "1")
    o, g = make_oracle(mech, seed=13, quirks=QUIRKS_FIXED, grid=_grid(), tlo=1100.0, thi=2600.0, radicals=1e-4)
    out = []
    for q in (0, 1):
        d = gpu.DeviceFlowfield(mech, g, quirks=QUIRKS_FIXED, flux_bits=64)
        d.upload_state(o)
        d.upload("RHS", np.zeros(d.shape("RHS")))
        d.set_elements(S.atoms_matrix(mech))
        d.set_tuning(adapt_queue=q)
        d.dt = 3e-8
        d.react_adaptive()
        out.append((d.status()["substeps"], {f: interior(d.download(f)) for f in ("CS", "T", "P")}))
        d.close()
    assert out[0][0] == out[1][0] > 33 * 5 * 3
    for f, v in out[0][1].items():
        assert rel_err(out[1][1][f], v) < TOL_FN, f


def test_imex_of_a_thin_gas(mech):
    o = Oracle(mech, _grid(), QUIRKS_FIXED)
    fill_state(o, 6, 1100.0, 1500.0)
    o.view("P")[:20] *= 2.0 ** -103
    o.prims_from_state()
    d = gpu.DeviceFlowfield(mech, _grid(), quirks=QUIRKS_FIXED, flux_bits=64)
    d.upload_state(o)
    o.update_after_cs()
    d.update_after_cs()
    D = interior(o.view("D"))
    assert (D < 1e-30).any() and (D > 1e-30).any()
    o.partial_t()
    o.dt = d.dt = 1e-12
    o.imex()
    d.imex()
    a, b = interior(d.download("CS")), interior(o.view("CS"))
    for part in (slice(0, 18), slice(18, None)):  # thin rows and the others, each to its own scale
        assert rel_err(a[part], b[part]) < TOL_FN
    assert rel_err(interior(d.download("T")), interior(o.view("T"))) < TOL_FN
    d.close()


def test_another_mechanism_may_take_a_denominator_past_the_range(mech):
    m = copy.deepcopy(mech)
    m.af[1] = 1e290  # H + O2 -> O + OH
    o = Oracle(m, _grid(), QUIRKS_FIXED)
    fill_state(o, 6, 1100.0, 1500.0)
    cs = o.view("CS")
    for s in ("O", "OH", "HO2", "H2O2", "H2O", "H2"):
        cs[..., m.species.index(s)] = 0.0
    cs[..., m.species.index("H")] = 1e-300
    d = gpu.DeviceFlowfield(m, _grid(), quirks=QUIRKS_FIXED, flux_bits=64)
    d.upload_state(o)
    o.update_after_cs()
    d.update_after_cs()
    o.view("RHS")[...] = 0.0
    d.upload("RHS", np.zeros(d.shape("RHS")))
    o.partial_t()
    o.dt = d.dt = 1e30
    with np.errstate(all="ignore"):
        o.imex()
        den = 1.0 - o.dt * interior(o.view("MDd"))[..., m.species.index("H")]
    d.imex()
    a, b = interior(d.download("CS")), interior(o.view("CS"))
    assert np.isinf(den).all() and np.isfinite(b).all() and (b[..., m.species.index("H")] == 1e-300).all()
    assert rel_err(a, b) < TOL_FN
    d.close()
