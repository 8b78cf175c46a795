"""A network's dataset and weights change between calls that keep its buffers:
each call works on its own rows and on the weights set last.  The first loss of
a training call is that of the weights before it on the call's first batch (all
rows in some order when the batch holds them), so it equals, to the order of
its sums, the loss that a fresh network reports for the same weights and rows.
"""
import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [128, 4096])
def test_each_training_call_reads_its_own_rows_and_weights(rows):
    import pticm
    rng = np.random.default_rng(rows)
    net = pticm.MLP(seed=1, batch=rows)
    for k in range(6):
        p = MO.init_like_device(k).astype(np.float32)
        X = rng.standard_normal((rows, MO.IN)).astype(np.float32)
        y = (rng.standard_normal(rows) + 3.0 * k).astype(np.float32)
        net.params = p
        first = net.train(X, y, 1, lr=1e-3, seed=k)[0]
        fresh = pticm.MLP(seed=2, batch=rows)
        fresh.params = p
        want, _ = fresh.gradients(X, y)
        # rows / 128 tile sums of 128 squares each, in another order: rows x 2^-24 relative at most
        assert abs(first - want) <= rows * 2.0 ** -24 * want, (k, first, want)


def test_predictions_in_portions():
    """More rows than one portion holds: each row's result is that of any other call, and device memory stays bounded."""
    torch = pytest.importorskip("torch")
    import pticm
    net = pticm.MLP(seed=1, batch=256)
    net.params = MO.init_like_device(3).astype(np.float32)
    part, n = 4 << 20, (4 << 20) + 777
    X = np.random.default_rng(0).standard_normal((n, MO.IN), dtype=np.float32)
    small = net.predict(X[part - 100:])
    before = torch.cuda.mem_get_info()[0]
    y = net.predict(X)
    assert before - torch.cuda.mem_get_info()[0] <= part * 32 + (8 << 20)   # (allocations come in 2 MB pieces)
    assert np.array_equal(y[part - 100:], small)
    assert np.array_equal(y[:1000], net.predict(X[:1000]))
