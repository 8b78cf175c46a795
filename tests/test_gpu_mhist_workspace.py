"""The multihistogram's device workspace: many instances whose matrix does not
fit shared memory share as many slots as run at once, take turns in fewer
slots with the same results, and without any are solved in the log domain.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNT, NT = 200, 96   # more instances than the GPU has SMs


def _batch():
    import pticm
    probs = []
    for k in range(COUNT):
        rng = np.random.default_rng(k)
        n = 420 + 3 * (k % 11)
        a = np.unique(np.sort(rng.integers(0, n, size=(2600, 2)), 1), axis=0)
        a = rng.permutation(a[a[:, 0] != a[:, 1]])[:2000]
        probs.append(pticm.Problem.from_coo(n, a[:, 0], a[:, 1], rng.choice([-1.0, 1.0], len(a))))
    b = pticm.Batch(probs, nt=NT, chains=1, seed=3, icm=False, exchange=0)
    b.set_ladders(np.linspace(1 / 0.5, 1 / 6.0, NT))
    b.init_states(4)
    b.enable_energy_histograms(30)
    b.run(130)
    return b


def test_workspace_is_bounded_and_changes_no_result():
    b = _batch()
    used = b.compute_logdos()
    full = [b.logdos(i) for i in range(COUNT)]
    # a slice: K (NT | 1 doubles a bin), counts, weights, shifts and ranges
    slices = np.array([len(d) for d, _, _ in full]) * ((NT | 1) * 8 + 32)
    slot = (slices.max() + 127) // 128 * 128
    assert slices.max() > 200 * 1024, "the instances have to outgrow shared memory"
    assert used % slot == 0 and 0 < used < COUNT * slot
    # four slots, then one however small the bound
    for most, slots in ((4 * slot, 4), (1, 1)):
        assert b.compute_logdos(max_workspace=int(most)) == slots * slot
        for i in range(COUNT):
            d, lo, it = b.logdos(i)
            assert it == full[i][2] and lo == full[i][1] and np.array_equal(d, full[i][0])
    assert b.compute_logdos(max_workspace=0) == 0
    for i in range(COUNT):
        d, lo, it = b.logdos(i)
        want = full[i][0]
        ok = want > -1e300
        # both round exponents of up to a few thousand nats (1e-12) over up to a thousand iterations
        assert it == full[i][2] and lo == full[i][1] and np.array_equal(ok, d > -1e300)
        assert np.abs(d[ok] - want[ok]).max() <= 1e-9 * np.abs(want[ok]).max()
