"""The narrow block team's gathered sweep: fields, energies and best states
after runs stay exact (a from-scratch recompute), in the layouts where the
threads of a site, the portions of a class and the lists' 16-byte pieces
change, next to the stored-field sweep past its degree line.  With and without
ICM the run from the same states and seed takes the same path (the random
stream of a site does not depend on how its field is found), so the
exchange-free, ICM-free part is compared state for state.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, deg, seed, h):
    import pticm
    rng = np.random.default_rng(seed)
    keys = np.unique(np.concatenate([np.minimum(a, b) * n + np.maximum(a, b) for a, b in
                                     [(rng.integers(0, n, 3 * n * deg), rng.integers(0, n, 3 * n * deg))]]))
    keys = keys[keys // n != keys % n]
    keys = rng.permutation(keys)[:max(1, n * deg // 2)]
    w = rng.choice([-2.0, -1.0, 1.0, 3.0], size=len(keys))
    return pticm.Problem.from_coo(n, keys // n, keys % n, w, rng.integers(-2, 3, n).astype(float) if h else None)


@pytest.mark.parametrize("n,deg", [(2, 1), (5, 2), (33, 3), (129, 8), (100, 40), (250, 38), (700, 9), (3500, 8), (5000, 6)])
@pytest.mark.parametrize("sweeps", [1, 2])
def test_fields_and_energies_stay_exact(n, deg, sweeps):
    import pticm
    p = _problem(n, deg, n, n % 2 == 1)
    for icm in (True, False):
        ctx = pticm.Context(p, nt=6, seed=3, sweeps=sweeps, icm=icm)
        ctx.set_ladder(pticm.beta_linspace(0.5, 4.0, 6))
        ctx.init_states(5)
        for steps in (1, 7):
            ctx.run(steps)
            assert ctx.verify() == 0
        s, E, _, _ = ctx.replicas()
        Eo, _ = p.evaluate(s)
        assert np.array_equal(Eo.astype(np.int64), E)


@pytest.mark.parametrize("n,deg", [(60, 14), (300, 20), (1000, 12), (2000, 20)])
def test_gathered_and_stored_fields_take_the_same_path(n, deg):
    """Between the degree lines an ICM context keeps stored fields and an ICM-free one gathers."""
    import pticm
    p = _problem(n, deg, n + 1, True)
    out = []
    for icm in (True, False):
        ctx = pticm.Context(p, nt=6, seed=3, icm=icm)
        ctx.set_ladder(pticm.beta_linspace(0.5, 4.0, 6), nc=3 if icm else 0)
        ctx.init_states(5)
        ctx.run(30, pticm.PHASE_SWEEP | pticm.PHASE_EXCHANGE)
        out.append(ctx.replicas())
        assert ctx.verify() == 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)
