"""Reading replicas back in portions: more rows than the export buffer holds come
out as they are, and the context keeps no more than that buffer.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_many_rows_are_read_in_portions():
    torch = pytest.importorskip("torch")
    import pticm
    n, nt = 120000, 128   # 256 replicas: 154 MB of states and fields
    i = np.arange(n)
    p = pticm.Problem.from_coo(n, i, (i + 1) % n, np.where(i % 3 == 0, 1.0, -1.0))
    ctx = pticm.Context(p, nt=nt, seed=3, icm=False)
    ctx.set_ladder(pticm.beta_linspace(0.5, 3.0, nt))
    ctx.init_states(5)
    ctx.run(3)
    before = torch.cuda.mem_get_info()[0]
    s, E, f, _ = ctx.replicas()
    assert before - torch.cuda.mem_get_info()[0] <= (64 << 20) + (4 << 20)   # (allocations come in 2 MB pieces)
    sp = 2 * s.astype(np.int32) - 1
    w = np.where(i % 3 == 0, 1, -1)
    assert np.array_equal(f, w * np.roll(sp, -1, 1) + np.roll(w * sp, 1, 1))
    assert np.array_equal((w * sp * np.roll(sp, -1, 1)).sum(1), E)
