"""Words read across blocks before they have arrived: a block whose partner's
spins are held back past its energies sees words of an earlier step, makes the
pass again until the step's have come, and the run takes the path it takes
without the delay, in every form of the cluster search and block layout; past the
wait limit it ends with an error status, and the context runs on.
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NT = 6


def _context(n, deg, **kw):
    import pticm
    rng = np.random.default_rng(n)
    a = np.unique(np.sort(rng.integers(0, n, size=(3 * n * deg, 2)), 1), axis=0)
    a = rng.permutation(a[a[:, 0] != a[:, 1]])[:n * deg // 2]
    h = rng.integers(-2, 3, n).astype(float) if n % 2 else None
    p = pticm.Problem.from_coo(n, a[:, 0], a[:, 1], rng.choice([-1.0, 1.0], len(a)), h)
    ctx = pticm.Context(p, nt=NT, seed=3, icm=True, **kw)
    ctx.set_ladder(pticm.beta_linspace(0.5, 3.0, NT), nc=NT)
    ctx.init_states(5)
    return ctx


LAYOUTS = {
    "narrow": (200, 6, {}),
    "narrow_linear": (333, 20, {}),
    "wide": (400, 6, dict(block_threads=1024)),
    "breadth_first": (300, 6, dict(icm_algo=1)),
    "labels": (300, 6, dict(icm_algo=3)),
    "warp_teams": (201, 6, dict(replicas_per_block=2)),
    "block_team_of_three": (900, 6, dict(replicas_per_block=3)),
    "spins_only": (60000, 6, dict(replicas_per_block=1)),
    "scratch_in_device_memory_2": (45001, 6, dict(replicas_per_block=2)),
    "scratch_in_device_memory_4": (40000, 6, dict(replicas_per_block=4)),
    # (the cluster search's scratch fits beside the spins: every pair is worked out once)
    "shared_pairs": (20001, 6, dict(replicas_per_block=2)),
    "shared_pairs_interleaved": (14016, 6, dict(replicas_per_block=4)),
}


@pytest.mark.parametrize("name", list(LAYOUTS))
def test_late_words_change_nothing(name):
    n, deg, kw = LAYOUTS[name]
    out = []
    for delay in (0, 30000, 400000):
        ctx = _context(n, deg, **kw)
        ctx.run(2)
        assert ctx.layout().blocks > 1
        ctx.set_publish_delay(delay)
        ctx.run(12)
        assert ctx.verify() == 0
        out.append(ctx.replicas())
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("name", ["narrow", "warp_teams"])
def test_words_that_stay_away_end_the_run(name):
    import pticm
    n, deg, kw = LAYOUTS[name]
    ctx = _context(n, deg, **kw)
    ctx.run(2)
    # (the held-back blocks' energies come at once, their spins 40 ms later)
    ctx.set_wait_limit(limit_ns=1_000_000)
    ctx.set_publish_delay(40_000_000)
    t0 = time.time()
    with pytest.raises(pticm.PticmError) as e:
        ctx.run(4)
    assert e.value.code == 5 and "wait expired" in str(e.value)
    assert time.time() - t0 < 10.0
    ctx.set_wait_limit(0)
    ctx.set_publish_delay(0)
    ctx.run(5)
    assert ctx.verify() == 0


def test_the_limit_holds_where_a_pass_is_long():
    """A pass over 40000 sites takes tens of microseconds: the wait still ends at its limit, long before the words come."""
    import pticm
    ctx = _context(40000, 6, replicas_per_block=4, icm_algo=1)
    ctx.run(2)
    ctx.set_wait_limit(limit_ns=2_000_000)
    ctx.set_publish_delay(40_000_000)
    with pytest.raises(pticm.PticmError) as e:
        ctx.run(1)
    assert e.value.code == 5 and "wait expired at site 4" in str(e.value)


def test_a_run_that_ends_between_shared_pairs_leaves_exact_energies():
    """With pairs worked out once, a block may have taken over some of its replicas' results when another's never comes."""
    import pticm
    ctx = _context(14016, 6, replicas_per_block=4)
    ctx.set_ladder(pticm.beta_linspace(1.0, 1.01, NT), nc=NT)   # (close enough that replicas change places in every step)
    for trial in range(30):
        ctx.run(5)
        ctx.set_wait_limit(limit_ns=1_000_000)
        ctx.set_publish_delay(10_000_000)
        with pytest.raises(pticm.PticmError) as e:
            ctx.run(4)
        assert e.value.code == 5 and "wait expired" in str(e.value)
        assert ctx.verify() == 0, trial
        E, _, state, _ = ctx.best()
        assert ctx.problem.evaluate(state[None, :])[0][0] == E, trial
        ctx.set_wait_limit(0)
        ctx.set_publish_delay(0)
