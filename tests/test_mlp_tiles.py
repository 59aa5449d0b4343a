"""The training kernel's tiles and gradient slices at the sizes where they can
go wrong: one sample, one tile less or more a sample, and more tiles than one
launch writes slices for (1024)."""
import numpy as np
import pytest

from icempm_b200 import surrogate as sg
from oracle import mlp_oracle as mo


def _pairs(n):
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 6)).astype(np.float32)
    y = np.stack([np.tanh(x[:, 0] - x[:, 1]), x[:, 2] * 0.5, np.cos(x[:, 3])], 1).astype(np.float32)
    return x, y


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 127, 128, 129, 1024 * 128 + 1])
def test_gradient_slices(n):
    """Against the oracle with the same BF16 operands: a rounding that falls
    the other way after FP32 sums of another order moves an operand by 2^-8,
    through at most three products, so 3 * 2^-8 of the gradient's norm; the
    loss sees the forward products only."""
    x, y = _pairs(n)
    net = sg.init_net(3)
    sg.normalise(net, *_pairs(512))
    g, loss = sg.gradient(net, x, y)
    g_ref, loss_ref = mo.backward(net, x, y)
    assert abs(loss - loss_ref) <= 3 * 2 ** -8 * loss_ref
    for lo, hi in ((sg.OFF_W1, sg.OFF_B1), (sg.OFF_B1, sg.OFF_W2), (sg.OFF_W2, sg.OFF_B2), (sg.OFF_B2, sg.OFF_W3),
                   (sg.OFF_W3, sg.OFF_B3), (sg.OFF_B3, sg.OFF_XMU)):
        assert np.linalg.norm(g[lo:hi] - g_ref[lo:hi]) <= 3 * 2 ** -8 * np.linalg.norm(g_ref[lo:hi])
    assert np.all(g[sg.OFF_XMU:] == 0)


@pytest.mark.gpu
@pytest.mark.parametrize("tiles", [1, 9, 200])
def test_training_repeats_exactly(tiles):
    """Slices are added in a fixed order: two runs give the same bits (fewer
    slices than warps that add them, a remainder, more than SMs)."""
    x, y = _pairs(3000)
    runs = []
    for _ in range(2):
        net = sg.init_net(3)
        sg.normalise(net, x, y)
        loss = sg.train(net, x, y, steps=20, batch_tiles=tiles, lr=3e-3, seed=5)
        runs.append((net.copy(), np.array(loss)))
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
