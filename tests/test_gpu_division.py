"""The network's branch-free division against IEEE division, over the operands
that reach it (the guards in mlp_fused.cu), their ends and mantissas next to
all ones.  Markstein's method gives the IEEE quotient where the reciprocal it
starts from is correctly rounded, which it is unless the divisor's mantissa is
all ones; there it may be one unit in the last place off.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1 << 21


def _divide(a, b):
    import pticm
    q = np.zeros_like(a)
    ptr = [x.ctypes.data_as(C.c_void_p) for x in (a, b, q)]
    assert pticm.lib().pticm_mlp_division_probe(*ptr, len(a)) == 0
    return q


def _log_uniform(rng, lo, hi, n=N):
    """Magnitudes lo .. hi, one in eight with a mantissa next to all ones or zeros, both ends among them."""
    x = np.exp(rng.uniform(np.log(lo), np.log(hi), n)).astype(np.float32)
    bits = x.view(np.uint32)
    edge = rng.integers(0, 8, n) == 0
    low = rng.choice(np.array([0, 1, 2, 0x7FFFFD, 0x7FFFFE, 0x7FFFFF], np.uint32), n)
    x = np.where(edge, (bits & np.uint32(0xFF800000)) | low, bits).astype(np.uint32).view(np.float32)
    x = np.clip(x, np.float32(lo), np.float32(hi))
    x[:2] = lo, hi
    return x


def _check(a, b):
    q = _divide(a, b)
    want = a / b
    assert np.all(np.abs(want[want != 0]) >= np.finfo(np.float32).tiny)
    off = np.abs(q.view(np.int32).astype(np.int64) - want.view(np.int32))
    ones = (b.view(np.uint32) & np.uint32(0x7FFFFF)) == 0x7FFFFF
    assert off[~ones].max(initial=0) == 0
    assert off[ones].max(initial=0) <= 1


def _ends(rng, lo, hi):
    return np.concatenate([np.linspace(lo, hi, N // 2), rng.uniform(lo, hi, N // 2)]).astype(np.float32)


def test_silu():
    rng = np.random.default_rng(1)
    z = np.concatenate([_ends(rng, -60, 60), _log_uniform(rng, 1e-18, 1e18), -_log_uniform(rng, 1e-18, 60)])
    z = z[(z > -60) & (z < 1e18) & (np.abs(z) > 1e-18)]
    with np.errstate(over="ignore"):
        b = np.float32(1) + np.exp(-z)
    _check(z, b)
    _check(np.ones_like(b), b)


def test_sigmoid_divisors():
    rng = np.random.default_rng(2)
    b = _log_uniform(rng, 1.0, 1.2e26)
    _check(np.ones_like(b), b)


@pytest.mark.parametrize("lo,hi", [(0.1, 1.0), (0.001, 1.0)])
def test_adam_bias_corrections(lo, hi):
    rng = np.random.default_rng(3)
    a = _log_uniform(rng, 1e-20, 1e15)
    _check(a * rng.choice(np.array([-1, 1], np.float32), N), _log_uniform(rng, lo, hi))


def test_adam_steps():
    # x = lr m / c1 and y = sqrt(v / c2) + eps with lr in 1e-8 .. 1e8
    rng = np.random.default_rng(4)
    _check(_log_uniform(rng, 1e-28, 1e24), _log_uniform(rng, 1e-8, 1e9))
    _check(_log_uniform(rng, 1e-28, 1e-26), _log_uniform(rng, 1e8, 1e9))
    _check(_log_uniform(rng, 1e22, 1e24), _log_uniform(rng, 1e-8, 1e-7))
