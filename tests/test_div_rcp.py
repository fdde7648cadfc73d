"""The FP64 path's division by a quantity whose reciprocal is at hand
(div_rcp, csrc/gpu/numeric.cuh): q = RN(x r), then RN(q + RN(x - q y) r).
Evaluated here in exact rational arithmetic with each operation rounded to a
double once, it equals the correctly rounded x / y: for random significands,
for divisors and dividends at the ends of a binade (where the reciprocal's
rounding error is largest), over the exponents the step meets, and for a
reciprocal that is itself a rounded product of two (two ulps off), as the
sound-wave rows use it.  On the GPU the FP64 step built on it matches the
oracle (test_gpu_step.py, test_gpu_substeps.py)."""
from fractions import Fraction

import numpy as np
import pytest

N = 4000


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def div_rcp(x, y, r):
    q = x * r
    return _fma(_fma(-q, y, x), r, q)


@pytest.mark.parametrize("kind", ["random", "divisor_end", "both_ends", "range", "product_reciprocal"])
def test_div_rcp_is_the_correctly_rounded_quotient(kind):
    rng = np.random.default_rng(11)
    x, y = 1.0 + rng.random(N), 1.0 + rng.random(N)
    ends = lambda: np.where(rng.random(N) < 0.5, 2.0 - rng.integers(1, 4096, N) * 2.0 ** -52,
                            1.0 + rng.integers(0, 4096, N) * 2.0 ** -52)
    if kind in ("divisor_end", "both_ends"):
        y = ends()
    if kind == "both_ends":
        x = ends()
    if kind == "range":
        x = x * 2.0 ** rng.integers(-300, 300, N) * rng.choice([-1.0, 1.0], N)
        y = y * 2.0 ** rng.integers(-100, 100, N) * rng.choice([-1.0, 1.0], N)
    r = 1.0 / y
    if kind == "product_reciprocal":
        a, b = 1.0 + rng.random(N), 1.0 + rng.random(N)
        y, r = a * b, (1.0 / a) * (1.0 / b)
    for xi, yi, ri in zip(x.tolist(), y.tolist(), r.tolist()):
        assert div_rcp(xi, yi, ri) == xi / yi, (xi.hex(), yi.hex())
