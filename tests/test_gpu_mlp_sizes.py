"""The fused network kernels at the sizes where a tile or a ring can go wrong:
row counts around 128-row tiles (prediction), batches with a partly filled
last tile and of one tile (gradients), a training call past the index ring's
first chunk, and activations beyond the range of the branch-free division.
References: the numpy network with the kernels' BF16 roundings (1e-2 of a
block, as the other gradient tests; 2e-2 absolute of an O(1) output: four
layers of BF16 activations).
"""
import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu


def _net(batch, scale=1.0, seed=4):
    import pticm
    net = pticm.MLP(seed=1, batch=batch)
    p = (scale * MO.init_like_device(seed)).astype(np.float32)
    net.params = p
    return net, p


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000, 152 * 128 + 1])
def test_predict_rows(n):
    net, p = _net(256)
    X = np.random.default_rng(n).standard_normal((n, MO.IN)).astype(np.float32)
    want, _ = MO.forward(p.astype(np.float64), X, True)
    assert np.abs(net.predict(X) - want).max() <= 2e-2 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("batch,n", [(1, 1), (128, 100), (129, 129), (512, 400)])
def test_gradients_of_part_filled_tiles(batch, n):
    net, p = _net(batch)
    rng = np.random.default_rng(n)
    X, t = rng.standard_normal((n, MO.IN)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    loss, g = net.gradients(X, t)
    ol, og = MO.loss_and_grad(p.astype(np.float64), X, t, True)
    assert abs(loss - ol) <= 1e-3 * abs(ol)
    assert np.linalg.norm(g - og) <= 1e-2 * np.linalg.norm(og)


def test_large_activations():
    """Pre-activations past +-60 take the operator's division (silu -> 0 and v)."""
    net, p = _net(128, scale=6.0)
    X = np.random.default_rng(2).standard_normal((200, MO.IN)).astype(np.float32) * 20
    want, cache = MO.forward(p.astype(np.float64), X, True)
    assert min(z.min() for z in cache[1]) < -60
    assert np.abs(net.predict(X) - want).max() <= 2e-2 * np.abs(want).max()


def test_training_past_the_index_ring():
    """600 steps cross both chunks of the index ring; twice the same call gives the same weights, and the loss falls."""
    rng = np.random.default_rng(0)
    X = rng.standard_normal((900, MO.IN)).astype(np.float32)
    t = np.tanh(X[:, 0]) + 0.1 * X[:, 1]
    got = []
    for _ in range(2):
        net, _ = _net(128)
        losses = net.train(X, t, 600, lr=1e-3, seed=5)
        got.append(net.params)
        assert losses[-50:].mean() < 0.2 * losses[:5].mean()
    assert np.array_equal(got[0], got[1])
