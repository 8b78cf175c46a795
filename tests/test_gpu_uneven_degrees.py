"""Graphs with uneven degrees: which sweep and which cluster search they get
(both rules look at the longest lists beside the mean degree), and that the
search chosen finds the clusters a breadth-first search finds: the run from
the same states and seed takes the same path.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(L):
    i = np.arange(L * L)
    r, c = i // L, i % L
    return L * L, np.concatenate([np.stack([i, r * L + (c + 1) % L], 1), np.stack([i, (r + 1) % L * L + c], 1)])


def _hubs(L, count, length):
    """A lattice of even L and `count` more sites, each a neighbour of `length` sites of one sublattice."""
    n, e = _lattice(L)
    i = np.arange(n)
    even = i[(i // L + i % L) % 2 == 0]
    rng = np.random.default_rng(length)
    more = [np.stack([np.full(length, n + k), rng.choice(even, length, replace=False)], 1) for k in range(count)]
    return n + count, np.concatenate([e] + more)


def _attached(n, m):
    """Preferential attachment with m links per site."""
    rng = np.random.default_rng(n + m)
    ends, e = [0], []
    for v in range(1, n):
        for u in {ends[rng.integers(len(ends))] for _ in range(m)}:
            e.append((v, u))
            ends += [v, u]
    return n, np.array(e)


def _random(n, m):
    rng = np.random.default_rng(n + m)
    a = rng.integers(0, n, size=(4 * m, 2))
    a = np.unique(np.sort(a[a[:, 0] != a[:, 1]], 1), axis=0)
    return n, rng.permutation(a)[:m]


def _star(n):
    return n, np.stack([np.zeros(n - 1, np.int64), np.arange(1, n)], 1)


def _ring(n):
    i = np.arange(n)
    return n, np.stack([i, (i + 1) % n], 1)


def _context(graph, nt=6, **kw):
    import pticm
    n, e = graph
    w = np.random.default_rng(n).choice([-1.0, 1.0], len(e))
    p = pticm.Problem.from_coo(n, e[:, 0], e[:, 1], w)
    ctx = pticm.Context(p, nt=nt, seed=3, **kw)
    ctx.set_ladder(pticm.beta_linspace(0.5, 3.0, nt))
    ctx.init_states(5)
    return p, ctx


GRAPHS = {
    "lattice": (_lattice(20), True),
    "lattice_few_hubs": (_hubs(30, 4, 32), True),
    "lattice_many_hubs": (_hubs(20, 4, 40), False),
    "attached_1": (_attached(400, 1), False),
    "attached_2": (_attached(400, 2), False),
    "attached_2_large": (_attached(2400, 2), False),
    "star": (_star(700), False),
    "long_lists_outside": (_hubs(44, 8, 64), False),   # united by a warp each
    "lists_around_the_warp_line": (_hubs(44, 12, 17), False),
    "ring": (_ring(2501), True),
    "random_1000": (_random(1000, 1250), True),
    "random_2000": (_random(2000, 2500), False),
    "lattice_2500": (_lattice(50), True),
    "lattice_2601": (_lattice(51), False),
}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_cluster_search_of_uneven_graphs(name):
    graph, every = GRAPHS[name]
    out = []
    for algo in (0, 1):
        p, ctx = _context(graph, icm=True, icm_algo=algo)
        if algo == 0:
            assert p.info().ncolors <= 3   # (the rule's other condition holds)
            assert ctx.paths()[1] == every
        if algo == 1:
            assert not ctx.paths()[1]
        ctx.run(25)
        assert ctx.verify() == 0
        out.append(ctx.replicas())
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def _with_hubs(graph, count, length):
    """`count` sites of a graph with `length` more neighbours each."""
    n, e = graph
    rng = np.random.default_rng(length)
    more = [np.stack([np.full(length, k), rng.choice(np.arange(count, n), length, replace=False)], 1) for k in range(count)]
    return n, np.unique(np.sort(np.concatenate([e] + more), 1), axis=0)


FIELDS = {
    "lattice": (_lattice(20), True, True),
    "lattice_hub": (_hubs(20, 1, 180), False, False),
    "lattice_short_hub": (_hubs(20, 1, 40), True, True),
    "degree_8": (_random(1000, 4000), True, True),
    "degree_8_hub": (_with_hubs(_random(1000, 4000), 1, 600), False, False),
    "degree_8_hubs": (_with_hubs(_random(1000, 3000), 4, 200), False, False),
    "degree_20": (_random(1500, 15000), False, True),
    "degree_20_hub": (_with_hubs(_random(1500, 15000), 1, 1400), False, False),
    "degree_40_hub": (_with_hubs(_random(1000, 20000), 1, 300), True, True),
}


@pytest.mark.parametrize("icm", [True, False])
@pytest.mark.parametrize("name", list(FIELDS))
def test_fields_of_uneven_graphs(name, icm):
    graph, with_icm, without = FIELDS[name]
    p, ctx = _context(graph, icm=icm)
    assert (ctx.paths()[0] > 0) == (with_icm if icm else without)
    ctx.run(25)
    assert ctx.verify() == 0
    s, E, _, _ = ctx.replicas()
    assert np.array_equal(p.evaluate(s)[0].astype(np.int64), E)


@pytest.mark.parametrize("n,deg", [(60, 14), (300, 20), (1000, 12), (2000, 20)])
def test_between_the_degree_lines_the_two_sweeps_differ(n, deg):
    """Graphs of these sizes store fields with ICM and gather without it."""
    graph = _random(n, n * deg // 2)
    assert _context(graph, icm=True)[1].paths()[0] == 0
    assert _context(graph, icm=False)[1].paths()[0] > 0
