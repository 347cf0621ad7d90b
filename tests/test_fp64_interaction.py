"""The FP64 walk's far interaction (walk_ops.cuh, fp64_contrib), restated: root and
quotient from one float approximation of 1/sqrt(r2) by fused multiply-adds.
Both must be the correctly rounded results, as the reference's sqrt and
division are, with the approximation anywhere within its error bound, also for
squares next to the midpoint of two doubles."""
import math
from fractions import Fraction

import numpy as np
import pytest


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def root_and_quotient(r2, m, y):
    g, k = r2 * y, 0.5 * y
    e = fma(-g, k, 0.5)
    g, k = fma(g, e, g), fma(k, e, k)
    e = fma(-g, k, 0.5)
    g, k = fma(g, e, g), fma(k, e, k)
    r = fma(fma(-g, g, r2), k, g)
    inv = 2.0 * k
    q = m * inv
    q = fma(fma(-q, r, m), inv, q)
    return r, fma(fma(-q, r, m), inv, q)


@pytest.mark.parametrize("ulps", [-4, 0, 4])
def test_root_and_quotient_are_correctly_rounded(ulps):
    rng = np.random.default_rng(abs(ulps) + 1)
    for i in range(3000):
        if i % 3 == 0:    # a sum of squares of floats, as the walk's
            s = (rng.uniform(-1, 1, 3) * 10.0 ** rng.uniform(-4, 2)).astype(np.float32)
            r2 = float(s[0]) ** 2 + float(s[1]) ** 2 + float(s[2]) ** 2
        elif i % 3 == 1:  # the double nearest the square of a midpoint
            r = math.exp(rng.uniform(-10, 5))
            mid = Fraction(r) + Fraction(math.ulp(r)) / 2
            r2 = float(mid * mid)
        else:             # a perfect square
            f = float(np.float32(math.exp(rng.uniform(-10, 5))))
            r2 = f * f
        m = float(np.float32(math.exp(rng.uniform(-12, 8))))
        y0 = np.float32(1.0 / math.sqrt(float(np.float32(r2))))
        y = float((y0.view(np.uint32) + np.uint32(ulps & 0xFFFFFFFF)).view(np.float32))
        r, q = root_and_quotient(r2, m, y)
        assert r == math.sqrt(r2) and q == m / r, (r2.hex(), m.hex())
