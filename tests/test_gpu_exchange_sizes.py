"""The exchange in the reference's order where its bookkeeping changes: one
pair, 31 to 33 pairs (a second pair per lane), 63 to 65 (beyond the bit
masks), with one to four chains, against the serial restatement with the same
draws."""
import os

import numpy as np
import pytest

from test_gpu_exchange import G, initial_order, serial_reference_order

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chains", [1, 2, 3, 4])
@pytest.mark.parametrize("nt", [2, 3, 32, 33, 34, 64, 65, 66])
def test_reference_order_sizes(nt, chains):
    import pticm
    prob = pticm.Problem.load(os.path.join(G, "pmL6.gset"))
    seed = 77 + nt
    ctx = pticm.Context(prob, nt=nt, chains=chains, seed=seed, icm=False, exchange=0)
    beta = pticm.beta_linspace(0.4, 3.0, nt)
    ctx.set_ladder(beta)
    ctx.init_states(5)
    ctx.run(2, pticm.PHASE_SWEEP)
    E = ctx.replicas()[1]
    slot = [int(x) for x in ctx.ladder()[1]]
    order = list(initial_order(seed, nt)) if nt > 2 else [0]
    R = nt * chains
    att, suc, ambiguous = np.zeros(R, np.int64), np.zeros(R, np.int64), []
    for step in range(2, 6):
        ctx.run(1, pticm.PHASE_EXCHANGE)
        order = serial_reference_order(E, slot, order, beta, step, seed, nt, chains, att, suc, ambiguous)
    assert not ambiguous
    assert ctx.ladder()[1].tolist() == slot
    _, datt, dsuc = ctx.stats()
    assert datt.tolist() == att.tolist() and dsuc.tolist() == suc.tolist()
    assert ctx.exchange_order().tolist() == [int(x) for x in order]
