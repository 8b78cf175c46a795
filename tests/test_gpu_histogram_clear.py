"""A run that starts right after its histograms were made counts every step: the
clearing of a large histogram buffer (some 800 MB here) is over before the run's
own stream counts into it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NT, STEPS = 4, 12


def _problem(n, m):
    import pticm
    rng = np.random.default_rng(1)
    a = np.unique(np.sort(rng.integers(0, n, size=(3 * m, 2)), 1), axis=0)
    a = rng.permutation(a[a[:, 0] != a[:, 1]])[:m]
    return pticm.Problem.from_coo(n, a[:, 0], a[:, 1], rng.choice([-127.0, 127.0], m))


def test_context_counts_every_step():
    import pticm
    ctx = pticm.Context(_problem(2000, 200000), nt=NT, seed=3, icm=False)
    ctx.set_ladder(pticm.beta_linspace(500.0, 4000.0, NT))
    ctx.init_states(5)
    ctx.run(1)
    ctx.enable_energy_histograms(0)
    ctx.run(STEPS)
    h, _ = ctx.energy_histograms()
    assert h.nbytes > 500 << 20
    assert np.array_equal(h.sum(1), np.full(2 * NT, STEPS))


def test_batch_counts_every_step():
    import pticm
    p = _problem(4000, 60000)   # (its acceptance tables have to fit a block)
    count = 6
    b = pticm.Batch([p] * count, nt=NT, chains=1, seed=3, icm=False)
    b.set_ladders(pticm.beta_linspace(500.0, 4000.0, NT))
    b.init_states(5)
    b.run(1)
    b.enable_energy_histograms(0)
    b.run(STEPS)
    for i in range(count):
        assert np.array_equal(b.energy_histograms(i)[0].sum(1), np.full(NT, STEPS))
