"""Blocks of four replicas of an instance too large for stored fields: the
spins interleaved, four fields from one 32-bit sum of signed digits.  Energies,
fields and best states are checked against a from-scratch recomputation (all
integers: equality), at site counts around the 32-site groups and 16-byte
rows, with lists longer than the pieces loaded ahead, with fields beyond what
a digit holds (and next to it), and in blocks of two and three replicas, which keep
a row per replica.  A run in two halves equals the run in one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, deg, wmax, hub, seed):
    import pticm
    rng = np.random.default_rng(seed)
    a, b = rng.integers(0, n, n * deg // 2), rng.integers(0, n, n * deg // 2)
    if hub:
        a, b = np.concatenate([a, np.full(hub, n // 3)]), np.concatenate([b, rng.integers(0, n, hub)])
    keys = np.unique(np.minimum(a, b) * n + np.maximum(a, b))
    keys = keys[keys // n != keys % n]
    w = rng.integers(1, wmax + 1, len(keys)) * rng.choice([-1.0, 1.0], len(keys))
    return pticm.Problem.from_coo(n, keys // n, keys % n, w, rng.integers(-2, 3, n).astype(float) if seed % 2 else None)


@pytest.mark.parametrize("n,deg,wmax,hub,rpb", [
    (13001, 6, 1, 0, 4), (14015, 12, 1, 0, 4), (14032, 40, 1, 0, 4), (20003, 8, 1, 120, 4), (14001, 6, 1, 700, 4),
    (13024, 6, 100, 0, 4), (20000, 40, 1, 0, 3), (20001, 12, 1, 0, 2)])
def test_states_stay_exact(n, deg, wmax, hub, rpb):
    import pticm
    p = _problem(n, deg, wmax, hub, n)
    out = []
    for parts in ((6,), (2, 4)):
        ctx = pticm.Context(p, nt=2 * rpb, chains=2, seed=3, icm=True, replicas_per_block=rpb)
        ctx.set_ladder(pticm.beta_linspace(0.2, 3.0, 2 * rpb))
        ctx.init_states(5)
        assert ctx.layout().state_mode == 1 and ctx.layout().replicas_per_block == rpb
        for steps in parts:
            ctx.run(steps)
            assert ctx.verify() == 0
        s, E, _, _ = ctx.replicas()
        Eo, _ = p.evaluate(s)
        assert np.array_equal(Eo.astype(np.int64), E)
        bE, _, bs, _ = ctx.best()
        assert p.evaluate(bs[None, :])[0][0] == bE
        out.append((s, E, bE))
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n,deg,nt,chains,rpb,nc,h", [
    (13001, 6, 12, 2, 4, 12, True), (14015, 3, 8, 4, 4, 5, False), (16000, 20, 20, 2, 4, 1, True),
    (20001, 12, 9, 2, 3, 9, True), (19999, 6, 8, 4, 2, 6, False)])
def test_shared_pairs_equal_the_owners_own(n, deg, nt, chains, rpb, nc, h):
    """The cluster does not depend on the search: with the breadth-first search
    each owner (algo 1) works its pairs out, with union-find (2) the blocks share
    them."""
    import pticm
    p = _problem(n, deg, 1, 0, 2 * n + int(h))
    out = []
    for algo in (2, 1):
        ctx = pticm.Context(p, nt=nt, chains=chains, seed=3, icm=True, replicas_per_block=rpb, icm_algo=algo)
        ctx.set_ladder(pticm.beta_linspace(0.1, 2.0, nt), nc=nc)
        ctx.init_states(5)
        ctx.run(9)
        assert ctx.verify() == 0
        out.append(ctx.replicas())
    for a, b in zip(*out):
        assert np.array_equal(a, b)
