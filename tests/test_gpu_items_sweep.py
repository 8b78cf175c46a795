"""The sweep of blocks that hold several replicas: four (replica, site) items
per thread and round.  Fields, energies and best states equal a from-scratch
recomputation (integers: equality) where items per class are fewer than the
threads, end inside a round, or span several replicas of a warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,deg,rpb,threads", [
    (2, 1, 4, 32), (5, 4, 2, 32), (33, 32, 8, 64), (70, 3, 5, 64), (400, 4, 16, 512), (511, 6, 10, 128),
    (1025, 20, 5, 512), (3001, 10, 2, 256)])
@pytest.mark.parametrize("sweeps", [1, 3])
def test_states_stay_exact(n, deg, rpb, threads, sweeps):
    import pticm
    rng = np.random.default_rng(n)
    a, b = np.triu_indices(n, 1) if n < 64 else (rng.integers(0, n, n * deg // 2), rng.integers(0, n, n * deg // 2))
    keys = np.unique(np.minimum(a, b) * n + np.maximum(a, b))
    keys = keys[keys // n != keys % n]
    w = rng.choice([-2.0, -1.0, 1.0, 3.0], size=len(keys))
    p = pticm.Problem.from_coo(n, keys // n, keys % n, w, rng.integers(-2, 3, n).astype(float) if n % 2 else None)
    out = []
    for parts in ((8,), (3, 5)):
        ctx = pticm.Context(p, nt=rpb, chains=2, seed=3, icm=True, sweeps=sweeps, replicas_per_block=rpb,
                            block_threads=threads)
        ctx.set_ladder(pticm.beta_linspace(0.1, 3.0, rpb))
        ctx.init_states(5)
        assert ctx.layout().replicas_per_block == rpb and ctx.layout().threads == threads
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
