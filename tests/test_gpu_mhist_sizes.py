"""The multihistogram fixed point at the sizes where its launch changes: one
temperature, fewer and more temperatures than a block has threads, one CTA
and a cluster of them, a slice of bins that does not fit shared memory, bins
without samples, and a first step far from the result.  Against the same
iteration in numpy FP64; both round the exponents (up to a few thousand
nats, so 1e-12 absolute, over up to a thousand iterations) differently, which
bounds the difference by 1e-9 of ln g's scale.
"""
import math

import numpy as np
import pytest


def _numpy(count, e, beta, n):
    ok = count > 0
    lc, be, z, it = np.log(count[ok]), np.outer(beta, e[ok]), np.zeros(len(beta)), 0
    while True:
        a = (math.log(n) - z)[:, None] - be
        t = a.max(0)
        lg = lc - (t + np.log(np.exp(a - t).sum(0)))
        v = lg - be
        t = v.max(1)
        new = t + np.log(np.exp(v - t[:, None]).sum(1))
        it += 1
        q = (z - new) / new
        z = new
        if not (q * q).sum() > 1e-7:
            out = np.full(len(count), -np.inf)
            out[ok] = lg
            return out, z, it


CASES = {
    "one_temperature": dict(beta=[0.4], var=400, samples=4000, gap=1),
    "two": dict(beta=[0.5, 0.4], var=300, samples=4000, gap=1),
    "every_other_level": dict(beta=np.linspace(0.6, 0.2, 9), var=300, samples=8000, gap=2),
    "cluster": dict(beta=np.linspace(0.9, 0.3, 21), var=2500, samples=8000, gap=1),
    "many_temperatures": dict(beta=np.repeat([0.5, 0.45], 65), var=200, samples=300, gap=1),
    "more_than_threads": dict(beta=np.repeat([0.5, 0.45], 270), var=100, samples=1000, gap=1),
    "slice_in_device_memory": dict(beta=np.repeat([0.5, 0.49], 170), var=60000, samples=200, gap=1),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CASES))
def test_fixed_point_sizes(name):
    import pticm
    k = CASES[name]
    rng = np.random.default_rng(5)
    beta = np.asarray(k["beta"], np.float64)
    rows, off, length, emin, at, top = [], [], [], [], 0, -math.inf
    for b in beta:
        step = 2.0 * k["gap"]
        e = step * np.round(rng.normal(-b * k["var"], math.sqrt(k["var"]), k["samples"]) / step)
        row = np.bincount(((e - e.min()) / 2).astype(np.int64)).astype(np.uint32)
        rows.append(row), off.append(at), length.append(len(row)), emin.append(e.min())
        at += len(row)
        top = max(top, e.max())
    emin = np.array(emin)
    nb = int(math.ceil((top - emin.min()) / 2.0))
    count = np.zeros(nb)
    for row, lo in zip(rows, emin):
        i0 = int(round((lo - emin.min()) / 2))
        m = min(len(row), nb - i0)
        count[i0:i0 + m] += row[:m]
    n = int(rows[0].sum())
    dos, z, it = pticm.mhist_dos(np.concatenate(rows), off, length, beta, emin, 2.0, n, top)
    want, wz, wit = _numpy(count, emin.min() + 2.0 * np.arange(nb), beta, n)
    assert it == wit and len(dos) == nb
    assert np.array_equal(dos < -1e300, np.isinf(want))
    ok = np.isfinite(want)
    scale = max(np.abs(want[ok]).max(), np.abs(wz).max(), 1.0)
    assert np.abs(dos[ok] - want[ok]).max() <= 1e-9 * scale
    assert np.abs(z - wz).max() <= 1e-9 * scale
