"""Performance cases of the PT-ICM framework.

Each case is one call, or the short run of calls, that a user's program makes
through the package's public entry points, at sizes from the repository's own
configurations, tests and benchmark.  `listed()` gives the fixed cases,
`draw(rng)` more of the same ranges, `prepare` what the program holds before
the call, `run` one pass, `work` the bytes and operations a pass cannot do
without, and `exact` the 64-bit values of computed (not sampled) outputs.
"""
import math
import os
import sys

import numpy as np

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (_ROOT, os.path.join(_ROOT, "pt-icm_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import pticm  # noqa: E402


# ------------------------------------------------------------------- cases
def _pt(name, graph, n, m, weights, nt, chains, steps, burn, T0, T1, linear=False, sweeps=1, exchange=1):
    return dict(name=name, kind="pt", graph=graph, n=n, m=m, weights=weights, nt=nt, chains=chains, steps=steps,
                burn=burn, T0=T0, T1=T1, linear=linear, sweeps=sweeps, exchange=exchange)


def listed():
    return [
        # the smallest call: a 6 x 6 lattice for a few steps, all launch and latency
        _pt("pt_tiny", "lattice", 36, 72, "pm", 8, 2, 20, 20, 0.5, 3.0),
        # the +-J lattice workload, L = 20 and 32 temperatures: a lattice user's run
        _pt("pt_lattice20", "lattice", 400, 800, "pm", 32, 2, 1000, 500, 0.5, 3.0),
        # the headline: sparse MaxCut in the shape of a Gset file, 64 temperatures
        _pt("pt_gset2000", "random", 2000, 19990, "one", 64, 2, 600, 600, 0.5, 15.0),
        # linear terms, odd sizes, several sweeps a step and the reference's exchange order
        _pt("pt_linear777", "random", 777, 3111, "pm", 21, 2, 100, 50, 0.4, 4.0, linear=True, sweeps=3, exchange=0),
        # the large instance: 20000 spins, mean degree 40, 512 replicas
        _pt("pt_large20000", "random", 20000, 400000, "pm", 128, 4, 100, 20, 0.5, 9.5),
        # many uneven instances in one launch: half lattices, half random graphs
        dict(name="batch_mix", kind="batch", count=96, nt=32, rpb=16, steps=40, burn=20, T0=0.5, T1=3.0),
        # training data of the learned ladder: a batched pilot run and every instance's ln g(E)
        dict(name="pilot_records", kind="records", count=32, nt=32, burn=100, steps=300),
        # the multihistogram ladder (--preprocess): pilot run, ln g(E), acceptance walk
        dict(name="cae_ladder", kind="cae", n=400, m=1600, nt=24, T0=0.8, T1=4.0, samples=1000, burn=1000),
        # ln g(E) from histograms the caller already has
        dict(name="mhist_dos", kind="mhist", spins=1000, nt=33, samples=20000),
        # training the surrogate network, a short call at the production batch size
        dict(name="mlp_train", kind="train", rows=60000, batch=1024, steps=128),
        # the network over a ladder's energy levels, an odd number of rows
        dict(name="mlp_predict", kind="predict", rows=50001, batch=1024),
        # scoring many states of one problem: energy, cut and all single-flip changes
        dict(name="evaluate", kind="evaluate", n=2000, m=19990, count=2048, with_dE=True),
    ]


def _logu(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["pt", "pt", "pt", "pt", "batch", "records", "cae", "mhist", "train", "predict", "evaluate"])
    if kind == "pt":
        big = rng.random() < 0.2
        if rng.random() < 0.4 and not big:
            L = int(round(_logu(rng, 6, 50)))
            graph, n, m, weights = "lattice", L * L, 2 * L * L, "pm"
        else:
            n = int(round(_logu(rng, 5000, 20000))) if big else int(round(_logu(rng, 36, 5000)))
            m = max(8, min(n * (n - 1) // 4, int(n * _logu(rng, 3, 40) / 2)))
            graph, weights = "random", rng.choice(["one", "pm", "pm", "small"])
        chains = 2
        if n > 3000:   # one replica in each block, or four
            nt = rng.choice([8, 16, 32, 64])
            if rng.random() < 0.5:
                nt, chains = 128, 4
        else:
            nt = int(round(_logu(rng, 5, 64)))
        sweeps = rng.choice([1, 1, 1, 2])
        budget = _logu(rng, 2e5, 1e9)
        steps = int(min(1000, max(10, budget / (nt * chains * n * sweeps))))
        steps = max(1, min(steps, int(1.02e9 / (nt * chains * n * sweeps))))
        deg = 2.0 * m / n
        return {k: v for k, v in _pt("", graph, n, m, weights, nt, chains, steps, min(200, steps), round(rng.uniform(0.4, 0.8), 3),
                                     round(max(3.0, 1.5 * math.sqrt(deg)), 3), rng.random() < 0.25, sweeps,
                                     rng.choice([1, 1, 0])).items() if k != "name"}
    if kind == "batch":
        return dict(kind=kind, count=int(round(_logu(rng, 8, 96))), nt=rng.choice([16, 32]), rpb=rng.choice([8, 16]),
                    steps=rng.randint(10, 40), burn=10, T0=0.5, T1=3.0)
    if kind == "records":
        return dict(kind=kind, count=int(round(_logu(rng, 4, 32))), nt=rng.choice([16, 24, 32]), burn=50,
                    steps=rng.randint(100, 300))
    if kind == "cae":
        n = int(round(_logu(rng, 64, 400)))
        return dict(kind=kind, n=n, m=int(n * rng.uniform(1.5, 4)), nt=rng.randint(8, 24), T0=0.8, T1=4.0,
                    samples=rng.randint(500, 1000), burn=rng.randint(200, 1000))
    if kind == "mhist":
        return dict(kind=kind, spins=int(round(_logu(rng, 50, 1000))), nt=rng.randint(8, 33),
                    samples=rng.randint(2000, 20000))
    if kind == "train":
        return dict(kind=kind, rows=int(round(_logu(rng, 3000, 60000))), batch=rng.choice([200, 512, 1024]),
                    steps=rng.randint(16, 128))
    if kind == "predict":
        return dict(kind=kind, rows=int(round(_logu(rng, 50, 50000))), batch=rng.choice([256, 1024]))
    n = int(round(_logu(rng, 60, 2000)))
    return dict(kind="evaluate", n=n, m=min(n * (n - 1) // 4, int(n * rng.uniform(3, 20) / 2)),
                count=int(round(_logu(rng, 1, 2048))), with_dE=rng.random() < 0.6)


# ------------------------------------------------------------------ inputs
def _random_edges(rng, n, m):
    """m distinct unordered pairs of n sites, uniform."""
    keys = np.zeros(0, np.int64)
    while len(keys) < m:
        a = rng.integers(0, n, size=2 * m + 64)
        b = rng.integers(0, n, size=2 * m + 64)
        lo, hi = np.minimum(a, b), np.maximum(a, b)
        keys = np.unique(np.concatenate([keys, (lo * n + hi)[lo != hi]]))
    keys = rng.permutation(keys)[:m]
    return (keys // n).astype(np.int32), (keys % n).astype(np.int32)


def _lattice_edges(L):
    i = np.arange(L * L, dtype=np.int32)
    r, c = i // L, i % L
    return np.concatenate([i, i]), np.concatenate([r * L + (c + 1) % L, ((r + 1) % L) * L + c]).astype(np.int32)


def _weights(rng, m, weights):
    if weights == "one":
        return np.ones(m)
    if weights == "pm":
        return rng.choice(np.array([-1.0, 1.0]), size=m)
    return rng.choice(np.array([-3.0, -2.0, -1.0, 1.0, 2.0, 3.0]), size=m)


def _graph(rng, graph, n, m, weights, linear=False):
    src, dst = _lattice_edges(math.isqrt(n)) if graph == "lattice" else _random_edges(rng, n, m)
    w = _weights(rng, len(src), weights)
    h = rng.integers(-2, 3, size=n).astype(np.float64) if linear else None
    return src, dst, w, h


def _mixed_graphs(rng, count):
    """The uneven mix of the batched workload: lattices and +-1 random graphs in turn
    (the sizes by the count alone, the graphs from `rng`)."""
    out, sizes = [], np.random.default_rng(1000 + count)
    for i in range(count):
        if i % 2 == 0:
            L = int(sizes.choice([10, 20, 32, 50]))
            out.append((L * L,) + _graph(rng, "lattice", L * L, 2 * L * L, "pm"))
        else:
            n = int(round(math.exp(sizes.uniform(math.log(200), math.log(5000)))))
            out.append((n,) + _graph(rng, "random", n, int(round(n * sizes.uniform(3, 20) / 2)), "pm"))
    return out


def _ladder_graphs(rng, count):
    """Instances of the learned-ladder workload: smaller lattices and random graphs in turn
    (the sizes by the count alone, the graphs from `rng`)."""
    out, sizes = [], np.random.default_rng(5000 + count)
    for i in range(count):
        if i % 2 == 0:
            L = int(sizes.integers(6, 31))
            out.append((L * L,) + _graph(rng, "lattice", L * L, 2 * L * L, "pm"))
        else:
            n = int(round(math.exp(sizes.uniform(math.log(100), math.log(1000)))))
            m = min(n * (n - 1) // 4, int(round(n * sizes.uniform(3, 20) / 2)))
            out.append((n,) + _graph(rng, "random", n, m, "pm"))
    return out


def _histograms(rng, spins, nt, samples):
    """Energy histograms of `samples` draws per temperature from a Gaussian density
    of states, cut to the range each temperature visited (no bin in it empty)."""
    var = 4.0 * spins
    beta = np.linspace(1.0, 0.25, nt)
    rows, off, length, emin = [], [], [], []
    at = 0
    top = -math.inf
    for b in beta:
        e = 2.0 * np.round((rng.normal(-b * var, math.sqrt(var), samples)) / 2.0)
        lo, hi = e.min(), e.max()
        row = np.bincount(((e - lo) / 2).astype(np.int64)) + 1
        rows.append(row)
        off.append(at)
        length.append(len(row))
        emin.append(lo)
        at += len(row)
        top = max(top, hi)
    hist = np.concatenate(rows).astype(np.uint32)
    return dict(hist=hist, hist_off=np.array(off, np.uint64), hist_len=np.array(length, np.uint64), beta_hist=beta,
                emin=np.array(emin), estep=2.0, n=int(rows[0].sum()), max_emax=top)


_IN, _K0, _H = 7, 64, 256
_KIN = [_K0, _H, _H, _H]


def _params(rng):
    """Network parameters in the flat order W1 b1 .. W4 b4 w5 b5, He scaling."""
    parts = []
    for layer, k in enumerate(_KIN):
        w = rng.normal(0, math.sqrt(2.0 / (_IN if layer == 0 else _H)), (_H, k))
        if layer == 0:
            w[:, _IN:] = 0
        parts += [w.ravel(), rng.normal(0, 0.05, _H)]
    parts += [rng.normal(0, math.sqrt(1.0 / _H), _H), np.array([0.1])]
    return np.concatenate(parts).astype(np.float32)


def _rows(rng, rows):
    """Instance features and E/W, and a smooth entropy-like target."""
    k = max(1, rows // 200)
    f = np.stack([rng.uniform(0.35, 0.85, k), rng.uniform(0.4, 0.9, k), rng.uniform(0.15, 1.0, k),
                  rng.uniform(0.0, 0.45, k), rng.uniform(-0.1, 0.1, k), rng.uniform(0.95, 1.0, k)], 1)
    x = np.concatenate([np.repeat(f, -(-rows // k), 0)[:rows], rng.uniform(-0.8, 0.4, (rows, 1))], 1)
    x = rng.permutation(x).astype(np.float32)
    y = (-6.0 * x[:, 6] ** 4 + np.sin(3.0 * x[:, 6]) * x[:, 2] + 0.3 * x[:, 0]).astype(np.float32)
    return x, y


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "pt":
        src, dst, w, h = _graph(rng, case["graph"], case["n"], case["m"], case["weights"], case["linear"])
        p = pticm.Problem.from_coo(case["n"], src, dst, w, h)
        ctx = pticm.Context(p, nt=case["nt"], chains=case["chains"], seed=seed + 1, sweeps=case["sweeps"], icm=True,
                            exchange=case["exchange"])
        ctx.set_ladder(pticm.beta_linspace(case["T0"], case["T1"], case["nt"]))
        ctx.init_states(seed + 1)
        ctx.run(case["burn"])
        s["ctx"] = ctx
    elif kind in ("batch", "records"):
        graphs = (_mixed_graphs if kind == "batch" else _ladder_graphs)(rng, case["count"])
        probs = [pticm.Problem.from_coo(*g) for g in graphs]
        if kind == "batch":
            b = pticm.Batch(probs, nt=case["nt"], seed=seed + 1, icm=True, replicas_per_block=case["rpb"])
            b.set_ladders(pticm.beta_linspace(case["T0"], case["T1"], case["nt"]))
            b.init_states(seed + 2)
            b.run(case["burn"])
            s["batch"] = b
        else:
            ends = [max(3.0, 1.5 * math.sqrt(2.0 * len(g[1]) / g[0])) for g in graphs]
            s["ladders"] = np.array([np.linspace(1 / 0.5, 1 / t, case["nt"]) for t in ends])
            s["problems"] = probs
            s["levels"] = 1 + max(len(g[1]) for g in graphs)   # energy levels -W, -W+2 .. W of +-1 couplings
            s["seed"] = seed
    elif kind == "cae":
        src, dst, w, h = _graph(rng, "random", case["n"], case["m"], "pm")
        s["problem"] = pticm.Problem.from_coo(case["n"], src, dst, w, h)
        s["seed"] = seed
    elif kind == "mhist":
        s["hist"] = _histograms(rng, case["spins"], case["nt"], case["samples"])
    elif kind in ("train", "predict"):
        net = pticm.MLP(seed=seed, batch=case["batch"])
        s["params"] = _params(rng)
        net.params = s["params"]
        s["net"] = net
        s["x"], s["y"] = _rows(rng, case["rows"])
        s["seed"] = seed
    else:
        src, dst, w, h = _graph(rng, "random", case["n"], case["m"], "one")
        s["problem"] = pticm.Problem.from_coo(case["n"], src, dst, w, h)
        s["states"] = rng.integers(0, 2, size=(case["count"], case["n"]), dtype=np.uint8)
    return s


# --------------------------------------------------------------------- run
def _table(ln_g, width):
    """ln g as a row of a table of all levels, levels without samples 0."""
    out = np.zeros(width)
    out[:len(ln_g)] = np.where(ln_g > -1e300, ln_g, 0.0)
    return out


def _mhist_width(case):
    return int(1.5 * case["spins"] + 40 * math.sqrt(case["spins"]))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "pt":
        ctx = s["ctx"]
        ctx.run(case["steps"])
        st, attempts, successes = ctx.stats()
        energy, sweep, state, replica = ctx.best()
        spins, E, fields, slot = ctx.replicas()
        return dict(flips=st.flips, swaps=st.swaps, attempts=attempts, successes=successes, best_energy=energy,
                    best_sweep=sweep, best_state=state, best_replica=replica, spins=spins, energies=E, fields=fields,
                    slots=slot)
    if kind == "batch":
        b = s["batch"]
        b.run(case["steps"])
        best, flips = b.best()
        energies = [b.energies(i) for i in range(case["count"])]
        return dict(best=best, flips=flips, energies=np.stack([e for e, _ in energies]),
                    slots=np.stack([k for _, k in energies]),
                    swaps=np.stack([b.swap_stats(i)[1] for i in range(case["count"])]),
                    states=np.concatenate([b.best_state(i) for i in range(case["count"])]))
    if kind == "records":
        b = pticm.Batch(s["problems"], nt=case["nt"], chains=1, seed=s["seed"] + 1, icm=False, exchange=0)
        b.set_ladders(s["ladders"])
        b.init_states(s["seed"] + 2)
        b.enable_energy_histograms(case["burn"])
        b.run(case["burn"] + case["steps"])
        b.compute_logdos()
        got = [b.logdos(i) for i in range(case["count"])]
        return dict(ln_g=np.stack([_table(d, s["levels"]) for d, _, _ in got]), emin=np.array([e for _, e, _ in got]),
                    iterations=np.array([it for _, _, it in got]))
    if kind == "cae":
        return pticm.cae_ladder(s["problem"], seed=s["seed"], T0=case["T0"], T1=case["T1"], nt=case["nt"],
                                samples=case["samples"], burn_in=case["burn"])
    if kind == "mhist":
        ln_g, ln_z, iterations = pticm.mhist_dos(**s["hist"])
        return _table(ln_g, _mhist_width(case)), ln_z, iterations
    if kind == "train":
        s["net"].params = s["params"]
        losses = s["net"].train(s["x"], s["y"], case["steps"], lr=1e-3, seed=s["seed"])
        return losses, s["net"].params
    if kind == "predict":
        return s["net"].predict(s["x"])
    return s["problem"].evaluate(s["states"], with_dE=case["with_dE"])


# -------------------------------------------------------------------- work
_NET = _H * (_K0 + 3 * _H) + _H   # weights of the network


def work(case):
    kind = case["kind"]
    if kind == "pt":
        R = case["nt"] * case["chains"]
        n, m = case["n"], case["m"]
        # spins in and out, fields out, the packed graph; four operations per attempted flip
        return {"bytes": 6 * R * n + 8 * m + 4 * n + n, "flops": 4 * case["steps"] * case["sweeps"] * R * n}
    if kind == "batch":
        n, m, R = 1200.0, 5000.0, 2 * case["nt"]   # mean sizes of the mix
        return {"bytes": case["count"] * (2 * R * n + 8 * m), "flops": 4 * case["count"] * case["steps"] * R * n}
    if kind == "records":
        n, m, R = 380.0, 1500.0, case["nt"]
        return {"bytes": case["count"] * (8 * m + R * 200 * 4 + 800 * 8),
                "flops": 4 * case["count"] * (case["burn"] + case["steps"]) * R * n}
    if kind == "cae":
        return {"bytes": 8 * case["m"] + case["nt"] * 8,
                "flops": 4 * (case["samples"] + case["burn"]) * case["nt"] * case["n"]}
    if kind == "mhist":
        bins, width = 3 * case["spins"] + 8 * math.sqrt(case["spins"]), 8 * math.sqrt(case["spins"])
        # about a thousand iterations, in each one multiply-add per visited (bin, temperature) and sum
        return {"bytes": case["nt"] * width * 4 + bins * 8, "flops": 4 * 1000 * case["nt"] * width}
    if kind == "train":
        return {"bytes": case["rows"] * 32 + 8 * _NET,
                "flops": 6 * case["steps"] * min(case["batch"], case["rows"]) * _NET}
    if kind == "predict":
        return {"bytes": case["rows"] * 32 + 4 * _NET, "flops": 2 * case["rows"] * _NET}
    n, c = case["n"], case["count"]
    return {"bytes": c * n * (9 if case["with_dE"] else 1) + 16 * c + 8 * case["m"], "flops": 4 * c * case["m"]}


# ------------------------------------------------------------------- exact
def _unpack(p):
    out, at = [], 0
    for k in _KIN:
        out.append((p[at:at + _H * k].reshape(_H, k), p[at + _H * k:at + _H * k + _H]))
        at += _H * k + _H
    return out, p[at:at + _H], p[at + _H:at + _H + 1]


def _forward(p, x):
    layers, w5, b5 = _unpack(p)
    h = np.zeros((len(x), _K0))
    h[:, :_IN] = x
    ins, sig = [], []
    for w, b in layers:
        z = h @ w.T + b
        sg = 1.0 / (1.0 + np.exp(-z))
        ins.append(h)
        sig.append((z, sg))
        h = z * sg
    return h @ w5 + b5[0], ins, sig, h


def _train_exact(p, x, y, batch, steps, lr, seed):
    """Adam over epoch-wise shuffled batches (xorshift64 Fisher-Yates), in 64 bits."""
    mask = (1 << 64) - 1
    n = len(x)
    order = list(range(n))
    g = (seed ^ 0xA0761D6478BD642F) & mask
    cursor = n
    nb = min(n, (batch + 127) // 128 * 128)
    m1, m2, losses = np.zeros_like(p), np.zeros_like(p), []
    for k in range(1, steps + 1):
        rows = []
        while len(rows) < nb:
            if cursor == n:
                for i in range(n - 1, 0, -1):
                    g ^= (g << 13) & mask
                    g ^= g >> 7
                    g ^= (g << 17) & mask
                    j = g % (i + 1)
                    order[i], order[j] = order[j], order[i]
                cursor = 0
            take = min(nb - len(rows), n - cursor)
            rows += order[cursor:cursor + take]
            cursor += take
        layers, w5, _ = _unpack(p)
        out, ins, sig, h4 = _forward(p, x[rows])
        e = out - y[rows]
        losses.append((e * e).mean())
        dy = 2.0 * e / nb
        grads = [h4.T @ dy, np.array([dy.sum()])]
        dh = dy[:, None] * w5
        for layer in range(3, -1, -1):
            z, sg = sig[layer]
            dz = dh * (sg * (1.0 + z * (1.0 - sg)))
            grads = [(dz.T @ ins[layer]).ravel(), dz.sum(0)] + grads
            dh = dz @ layers[layer][0] if layer else None
        gr = np.concatenate(grads)
        m1 = 0.9 * m1 + 0.1 * gr
        m2 = 0.999 * m2 + 0.001 * gr * gr
        p = p - lr * (m1 / (1 - 0.9 ** k)) / (np.sqrt(m2 / (1 - 0.999 ** k)) + 1e-8)
    return np.array(losses), p


def _mhist_exact(hist, hist_off, hist_len, beta_hist, emin, estep, n, max_emax):
    """The multihistogram fixed point in 64 bits, to the same stopping rule."""
    lo = emin.min()
    nb = int(math.ceil((max_emax - lo) / estep))
    e = lo + estep * np.arange(nb)
    count = np.zeros(nb)
    for o, k, b in zip(hist_off.astype(int), hist_len.astype(int), emin):
        i0 = int(round((b - lo) / estep))
        k = min(k, nb - i0)
        count[i0:i0 + k] += hist[o:o + k]
    lc = np.log(count)
    z = np.zeros(len(beta_hist))
    be = np.outer(beta_hist, e)
    it = 0
    while True:
        a = (math.log(n) - z)[:, None] - be
        top = a.max(0)
        lg = lc - (top + np.log(np.exp(a - top).sum(0)))
        v = lg - be
        top = v.max(1)
        new = top + np.log(np.exp(v - top[:, None]).sum(1))
        it += 1
        q = (z - new) / new
        z = new
        if not (q * q).sum() > 1e-7:
            return lg, z, it


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "mhist":
        ln_g, ln_z, it = _mhist_exact(**_histograms(rng, case["spins"], case["nt"], case["samples"]))
        return _table(ln_g, _mhist_width(case)), ln_z, it
    if kind in ("train", "predict"):
        p = _params(rng).astype(np.float64)
        x, y = _rows(rng, case["rows"])
        if kind == "predict":
            return _forward(p, x.astype(np.float64))[0]
        return _train_exact(p, x.astype(np.float64), y.astype(np.float64), case["batch"], case["steps"],
                            float(np.float32(1e-3)), seed)
    if kind == "evaluate":
        n = case["n"]
        src, dst, w, _ = _graph(rng, "random", n, case["m"], "one")
        spins = 2.0 * rng.integers(0, 2, size=(case["count"], n), dtype=np.uint8) - 1.0
        J = np.zeros((n, n))
        J[src, dst] = w
        J += J.T
        f = spins @ J
        E = 0.5 * (spins * f).sum(1)
        cut = 0.5 * (w.sum() - E)
        return (E, cut, -2.0 * spins * f) if case["with_dE"] else (E, cut)
    return None   # Markov-chain trajectories: whole numbers, equal or not
