"""Problems whose energies need more than 30 and more than 32 bits: cluster moves
sum their energy changes in 64 bits, and past 32 bits the blocks meet at the
counting barrier and exchange plain energies beside the tagged spin words.  A
complete bipartite graph with couplings of +-127 reaches both with few sites.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[2950, 4200])
def problem(request):
    import pticm
    a = request.param
    w = np.random.default_rng(a).choice([-127.0, 127.0], a * a)
    bound = 127 * a * a
    assert bound > (1 << 30 if a == 2950 else 1 << 31)
    return pticm.Problem.from_coo(2 * a, np.repeat(np.arange(a), a), a + np.tile(np.arange(a), a), w)


@pytest.mark.parametrize("rpb", [0, 1, 2, 4])
@pytest.mark.parametrize("exchange", [0, 1])
def test_energies_stay_exact(problem, rpb, exchange):
    import pticm
    ctx = pticm.Context(problem, nt=4, seed=3, icm=True, replicas_per_block=rpb, exchange=exchange)
    ctx.set_ladder(pticm.beta_linspace(1000.0, 20000.0, 4), nc=4)
    ctx.init_states(5)
    ctx.run(3)
    assert ctx.layout().blocks > 1
    assert ctx.verify() == 0
    s, E, _, _ = ctx.replicas()
    assert np.array_equal(problem.evaluate(s)[0].astype(np.int64), E)
