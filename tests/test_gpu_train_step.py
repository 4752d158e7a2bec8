"""The fused training step (one block per 128 samples, weight gradients kept on
chip over a block's samples) where its split changes: one tile per block, the
largest batch with one tile per block, and batches whose blocks take two tiles
-- with some blocks taking one more than others.

Tolerances: the repository's bars for the BF16 pipeline against the quantised
FP64 oracle (1.5 % of each parameter's gradient norm, 2e-3 of the loss, 2 % of
the output scale); only FP32 summation order depends on the batch.  The partial
sums are added in block order, so a repeated run has the same bits."""
import numpy as np
import pytest

from mlp_oracle import loss_grad, unpack

from _cases import QUIRKS_FIXED, small_grid
from eu3d_b200 import gpu
from eu3d_b200 import surrogate as S
from test_gpu_surrogate import LAYERS, _batch, _params, _rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(mech):
    d = gpu.DeviceFlowfield(mech, small_grid(), QUIRKS_FIXED, flux_bits=64)
    yield d
    d.close()


@pytest.mark.parametrize("B", [256, 18944, 19200, 37888 + 256])
def test_batch_split(dev, B):
    sur = gpu.DeviceSurrogate(dev, 0, S.atoms_matrix(dev.mech))
    p = _params(17)
    sur.set_params(p)
    X, Y = _batch(B, B)
    loss, g, out = sur.loss_grad(X, Y)
    loss_o, g_o, out_o = loss_grad(p.astype(np.float64), X.astype(np.float64), Y.astype(np.float64), quantize=True)
    assert abs(loss - loss_o) <= 2e-3 * loss_o
    assert np.max(np.abs(out[:, :10] - out_o[:, :10])) <= 2e-2 * np.max(np.abs(out_o[:, :10]))
    gd, god = unpack(g), unpack(g_o)
    for name in LAYERS:
        assert _rel(gd[name], god[name]) < 1.5e-2, (name, _rel(gd[name], god[name]))
    loss2, g2, out2 = sur.loss_grad(X, Y)
    assert loss2 == loss and np.array_equal(g, g2) and np.array_equal(out, out2)
    sur.close()


def test_training_repeats_bit_for_bit_and_follows_the_gradient(dev):
    """Two runs from the same weights and seed agree in every bit, whatever the
    steps are split into: the batch of a step depends on its number alone."""
    sur = gpu.DeviceSurrogate(dev, 4096, S.atoms_matrix(dev.mech))
    env = (900.0, 2500.0, np.log(0.5), np.log(20.0), np.log(1e-9), np.log(1e-8))
    sur.add_random(4096, env, S.species_index(dev.mech), 5)
    sur.label(gpu.REACT_ADAPTIVE)
    X, Lb = sur.dataset()
    sur.set_norm(S.make_norm(dev.mech, X, Lb, env=env))
    runs = []
    for chunks in ((40,), (40,), (7, 33)):
        sur.set_params(S.init_params(3))
        losses = np.concatenate([sur.train(n, 512, 1e-3, 1e-3, 0, 99) for n in chunks])
        runs.append((losses, sur.get_params()))
    for losses, params in runs[1:]:
        assert np.array_equal(losses, runs[0][0]) and np.array_equal(params, runs[0][1])
    assert runs[0][0][-5:].mean() < 0.9 * runs[0][0][:5].mean()
    sur.close()
