"""The cluster search that unites along every edge (few neighbours, few
colours, at most 2560 sites) and, past its size line, the sampled one: the
states after an ICM phase with given seeds against a plain flood fill, on
lattices with two and three colour classes, at both sides of the line, in
every block layout.  Sites are few enough to compare exactly.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NT = 4


def _cluster(adj, diff, seed):
    seen, todo = {seed}, [seed]
    while todo:
        for v in adj[todo.pop()]:
            if diff[v] and v not in seen:
                seen.add(v)
                todo.append(v)
    return np.fromiter(seen, np.int64)


@pytest.mark.parametrize("layout", [{}, dict(block_threads=1024), dict(replicas_per_block=2), dict(replicas_per_block=2 * NT)])
@pytest.mark.parametrize("L", [3, 7, 20, 50, 51])
def test_lattice_clusters(L, layout):
    import pticm
    from pticm import instances
    inst = instances.pm_lattice(L, seed=L)
    prob = pticm.Problem.from_instance(inst)
    n = inst.n
    adj = [[] for _ in range(n)]
    for u, v in zip(inst.src.tolist(), inst.dst.tolist()):
        adj[u].append(v)
        adj[v].append(u)
    rng = np.random.default_rng(L)
    S = rng.integers(0, 2, size=(2 * NT, n), dtype=np.uint8)
    for k, f in enumerate([0.1, 0.3, 0.45, 0.8]):
        S[NT + k] = S[k] ^ (rng.random(n) < f).astype(np.uint8)
    ctx = pticm.Context(prob, nt=NT, seed=3, icm=True, **layout)
    ctx.set_ladder(pticm.beta_linspace(0.5, 3.0, NT), nc=NT)
    ctx.set_states(S)
    seeds = np.full(NT, -2, np.int64)
    want = {}
    for q in range(NT):
        k = NT - 1 - q
        a, b = S[k].copy(), S[NT + k].copy()
        if (a != b).sum() > n // 2:
            a ^= 1
        diff = a != b
        if not diff.any():
            continue
        seeds[q] = rng.choice(np.nonzero(diff)[0])
        c = _cluster(adj, diff, int(seeds[q]))
        a[c] ^= 1
        b[c] ^= 1
        want[k] = (a, b, 2 * len(c) > diff.sum())
    ctx.icm_pairs(seeds)
    out = ctx.replicas()[0]
    for k, (a, b, swapped) in want.items():
        got = (out[NT + k], out[k]) if swapped else (out[k], out[NT + k])
        assert np.array_equal(got[0], a) and np.array_equal(got[1], b), k
    assert ctx.verify() == 0
