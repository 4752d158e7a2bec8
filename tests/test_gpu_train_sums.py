"""The order in which the training step sums a small batch's gradients.

One tensor-core accumulation per 256 rows and parameter, chunks added in
order; bias gradients summed over the chunks per row, then as a tree over the
256 rows.  golden/sur_grad_sums.npz holds gradients that an implementation with
one GEMM and one column sum per layer recorded on a B200: every 61st weight and
every bias at one and two chunks (where it repeated itself bit for bit), the
biases at three and fifteen (the largest batch of this order).  The inputs are
host arrays, so nothing but the step's own sums enters.  Equality is of bits:
another order of the same sums moves a run of 70 optimiser steps by 1e-4."""
import os

import numpy as np
import pytest

from _cases import QUIRKS_FIXED, small_grid
from eu3d_b200 import gpu
from eu3d_b200 import surrogate as S
from test_gpu_surrogate import _batch, _params

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "sur_grad_sums.npz")
BATCHES = (256, 512, 768, 3840)


def recorded_indices(B):
    bias = np.concatenate([np.arange(o, o + n) for o, n in (S.OFF[b] for b in ("b1", "b2", "b3", "b4"))])
    return np.union1d(bias, np.arange(0, S.NPARAM, 61)) if B <= 512 else bias


def gradient(mech, B):
    d = gpu.DeviceFlowfield(mech, small_grid(), QUIRKS_FIXED, flux_bits=64)
    sur = gpu.DeviceSurrogate(d, 0, S.atoms_matrix(mech))
    sur.set_params(_params(17))
    _, g, _ = sur.loss_grad(*_batch(B + 1, B))
    sur.close()
    d.close()
    return g[recorded_indices(B)]


@pytest.mark.parametrize("B", BATCHES)
def test_small_batch_sums_have_the_recorded_bits(mech, B):
    assert np.array_equal(gradient(mech, B), np.load(GOLDEN)[f"g{B}"])
