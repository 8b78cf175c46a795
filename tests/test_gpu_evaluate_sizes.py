"""State scoring where its path changes: one site to a block's width, states
with linear terms, the largest state whose energy changes fit shared memory
and the first that does not, more states than one portion; exact integers
against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count,with_dE", [(1, 3, True), (33, 1, True), (513, 7, True), (46000, 3, True), (46500, 3, True),
                                             (46500, 3, False), (2000, 4500, True)])
def test_evaluate_sizes(n, count, with_dE):
    import pticm
    rng = np.random.default_rng(n)
    m = 3 * n if n > 1 else 0
    src = rng.integers(0, n, m)
    dst = (src + 1 + rng.integers(0, max(n - 1, 1), m)) % n
    w = rng.integers(-3, 4, m).astype(float)
    h = rng.integers(-2, 3, n).astype(float)
    p = pticm.Problem.from_coo(n, src, dst, w, h)
    states = rng.integers(0, 2, size=(count, n), dtype=np.uint8)
    got = p.evaluate(states, with_dE=with_dE)
    for g in np.unique(np.linspace(0, count - 1, 12).astype(int)):
        s = 2 * states[g].astype(np.int64) - 1
        f = np.zeros(n, np.int64)
        np.add.at(f, src, w.astype(np.int64) * s[dst])
        np.add.at(f, dst, w.astype(np.int64) * s[src])
        assert got[0][g] == (h * s).sum() + (s * f).sum() / 2
        assert got[1][g] == w[s[src] != s[dst]].sum()
        if with_dE:
            assert np.array_equal(got[2][g], -2.0 * s * (h + f))
