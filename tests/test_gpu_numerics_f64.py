"""The FP64 path's quotient by a reciprocal at hand (div_rcp), its reciprocal
(rcp_full), halving (half_of) and powers (cube, fourth) as the device computes
them (game_gpu_numerics), against the device's IEEE operations and exact
rational arithmetic.

div_rcp must give IEEE x / y bit for bit, infinities, NaN, signed zeros,
subnormals and overflows included, where r is the correctly rounded reciprocal
of y.  Where r carries another ulp (rcp_nr<2>, a product of two reciprocals)
the last remainder can lie on the wrong side for a dividend whose quotient is as
near to the middle of two doubles as quotients come, which needs a divisor
near the end of its binade: there one ulp is allowed, for those divisors
alone.  cube and fourth round a sum of two doubles that carries the power to
some 2^-104: equal to the exact power rounded once.  div_sweep, the column
sweeps' form, gives IEEE's quotient for divisors of 0, infinite, NaN or normal
up to 2^1022 wherever the quotient is not subnormal and the dividend not below
2^-900."""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

from game_archived_gb300 import native

pytestmark = pytest.mark.gpu

N = 1 << 20
DIV_RCP, DIV_RCP_NR, DIV, DIV_PRODUCT, DIV_SQUARE, RCP_FULL, HALF_OF, HALF, CUBE, FOURTH, SWEEP = range(11, 22)


def _run(op, x, y=None):
    lib = native.gpu()
    a = np.ascontiguousarray(x if y is None else np.concatenate([x, y]))
    out = np.empty(len(x))
    rc = lib.game_gpu_numerics(op, a.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p), len(x))
    assert rc == 0, lib.game_gpu_last_error().decode()
    return out


def _doubles(rng, n, lo, hi):
    return rng.choice([-1.0, 1.0], n) * np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))


def _ends(rng, n):
    """significands at either end of a binade"""
    return np.where(rng.random(n) < 0.5, 2.0 - rng.integers(1, 4096, n) * 2.0 ** -52,
                    1.0 + rng.integers(0, 4096, n) * 2.0 ** -52) * np.ldexp(1.0, rng.integers(-20, 20, n))


def _specials():
    f = np.finfo(np.float64)
    v = [0.0, np.inf, np.nan, 1.0, 3.0, 0.1, f.max, f.tiny, f.smallest_subnormal, f.tiny / 3, 2.0 ** -1000, 2.0 ** 1000,
         2.0 ** -501, 2.0 ** 501, 1e-300, 1e300, 2.0 - 2.0 ** -52]
    v = np.array(v + [-a for a in v])
    return np.repeat(v, v.size), np.tile(v, v.size)


def _pairs(rng):
    sx, sy = _specials()
    x = [_doubles(rng, N, -60, 60), _doubles(rng, N, -520, 520), _doubles(rng, N, -1074, 1023), _ends(rng, N // 4), sx,
         np.zeros(64), -np.zeros(64)]
    y = [_doubles(rng, N, -60, 60), _doubles(rng, N, -520, 520), _doubles(rng, N, -1074, 1023), _ends(rng, N // 4), sy,
         _doubles(rng, 64, -60, 60), _doubles(rng, 64, -60, 60)]
    return np.concatenate(x), np.concatenate(y)


def _same(a, b):
    """equal bits, or NaN on both sides"""
    return (a.view(np.uint64) == b.view(np.uint64)) | (np.isnan(a) & np.isnan(b))


def _near_the_end(y):
    m, _ = np.frexp(np.abs(np.where(np.isfinite(y) & (y != 0), y, 1.0)))
    return m > 1.0 - 2.0 ** -30


def test_div_rcp_is_the_ieee_quotient():
    x, y = _pairs(np.random.default_rng(21))
    ok = _same(_run(DIV_RCP, x, y), _run(DIV, x, y))
    assert ok.all(), (x[~ok][:5], y[~ok][:5])
    with np.errstate(all="ignore"):
        ok = _same(_run(DIV, x, y), x / y)
    assert ok.all(), (x[~ok][:5], y[~ok][:5])


@pytest.mark.parametrize("op,ieee", [(DIV_RCP_NR, DIV), (DIV_PRODUCT, DIV_SQUARE)])
def test_div_rcp_with_an_inexact_reciprocal(op, ieee):
    x, y = _pairs(np.random.default_rng(22))
    a, b = _run(op, x, y), _run(ieee, x, y)
    bad = ~_same(a, b)
    with np.errstate(all="ignore"):
        divisor = y if op == DIV_RCP_NR else y * y
    assert not (bad & ~_near_the_end(divisor)).any(), (x[bad][:5], y[bad][:5])
    assert (np.abs(a.view(np.int64)[bad] - b.view(np.int64)[bad]) <= 1).all()


def test_rcp_full_is_the_ieee_reciprocal():
    x, y = _pairs(np.random.default_rng(23))
    a, b = _run(RCP_FULL, y), _run(DIV, np.ones_like(y), y)
    bad = ~_same(a, b)
    assert not (bad & ~_near_the_end(y)).any(), y[bad][:5]
    assert (np.abs(a.view(np.int64)[bad] - b.view(np.int64)[bad]) <= 1).all()


def test_div_sweep_in_its_domain():
    x, y = _pairs(np.random.default_rng(26))
    with np.errstate(all="ignore"):
        z = x / y
        tiny = np.finfo(np.float64).tiny
        domain = (((np.abs(y) >= tiny) & (np.abs(y) <= 2.0 ** 1022)) | (y == 0) | ~np.isfinite(y)) \
            & ((np.abs(x) >= 2.0 ** -900) | (x == 0) | np.isnan(x)) & ~((np.abs(z) < tiny) & (z != 0))
    x, y = x[domain], y[domain]
    a, b = _run(SWEEP, x, y), _run(DIV, x, y)
    bad = ~_same(a, b)
    assert not (bad & ~_near_the_end(y)).any(), (x[bad][:5], y[bad][:5], a[bad][:5], b[bad][:5])
    assert (np.abs(a.view(np.int64)[bad] - b.view(np.int64)[bad]) <= 1).all()


def test_half_of_is_the_exact_half():
    x = np.concatenate(_pairs(np.random.default_rng(24)))
    ok = _same(_run(HALF_OF, x), _run(HALF, x))
    assert ok.all(), x[~ok][:5]


@pytest.mark.parametrize("op,n", [(CUBE, 3), (FOURTH, 4)])
def test_powers_are_correctly_rounded(op, n):
    rng = np.random.default_rng(25)
    x = np.concatenate([rng.uniform(-40.0, 40.0, 20000), _doubles(rng, 4000, -60, 60), _ends(rng, 4000),
                        np.arange(-40.0, 41.0)])
    a = _run(op, x)
    for xi, ai in zip(x.tolist(), a.tolist()):
        assert ai == float(Fraction(xi) ** n), xi.hex()
