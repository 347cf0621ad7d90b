"""The cell moments' rounded quotient (tree_ops.cuh, quot_float), restated.

float(c / m), with the quotient first rounded to double, is taken from
q = c * r with r ~ 1/m good to 2^-44, unless q lies within 512 of its units of a
point M halfway between two floats; there rho = c - M m decides the side.  The
restatement must equal the plain double division rounded to float on ties,
on quotients a few double units from a tie and on generic ones, with the
reciprocal at both ends of its error bound.
"""
import struct
from fractions import Fraction

import numpy as np
import pytest


def _bits(d):
    return struct.unpack("<Q", struct.pack("<d", d))[0]


def _double(b):
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def quot_float(c, m, r):
    """(value, how): how is 'q', 'side', 'tie' or 'division'."""
    b = _bits(c * r)
    ex, rem = (b >> 52) & 0x7FF, b & 0x1FFFFFFF
    if not 1023 - 125 <= ex <= 1023 + 126:
        return np.float32(c / m), "division"
    if abs(rem - 0x10000000) > 512:
        return np.float32(c * r), "q"
    mid = (b & ~0x1FFFFFFF) | 0x10000000
    rho = float(Fraction(c) - Fraction(_double(mid)) * Fraction(m))
    far = _double(_bits(m) + ((ex - 1023 - 51) << 52))
    if rho != 0 and abs(rho) < far:
        return np.float32(c / m), "division"
    down = (mid & 0x7FFFFFFFFFFFFFFF) >> 29
    up = bool(down & 1) if rho == 0 else (rho < 0) == bool(mid >> 63)
    bits = (down - ((1023 - 127) << 23)) + int(up) | (mid >> 63) << 31
    return np.uint32(bits).view(np.float32), "tie" if rho == 0 else "side"


@pytest.mark.parametrize("error", [-(2.0 ** -44.5), 0.0, 2.0 ** -44.5])
def test_quotient_equals_division(error):
    rng = np.random.default_rng(20261205)
    seen = set()
    for i in range(6000):
        w = float(np.float32(np.exp(rng.uniform(-15, 10))))
        x = rng.uniform(-50, 100) + rng.uniform(-1, 1, size=2) * 10.0 ** rng.uniform(-6, 0)
        x = [float(v) for v in x.astype(np.float32)]
        m, c = 2 * w, x[0] * w + x[1] * w  # two equal masses: ties are common
        if i % 3 == 1:                     # close to a tie of a generic mass
            M = _double(_bits(x[0]) & ~0x1FFFFFFF | 0x10000000)
            m = w * (1.0 + int(rng.integers(1000)) * 2.0 ** -50)
            c = _double(_bits(M * m) + int(rng.integers(-12, 13)))
        elif i % 3 == 2:
            m, c = 3.7 * w, x[0] * w + x[1] * (2.7 * w)
        if c == 0:
            continue
        got, how = quot_float(c, m, (1.0 / m) * (1.0 + error))
        seen.add(how)
        want = np.float32(c / m)
        assert got.view(np.uint32) == want.view(np.uint32), (c.hex(), m.hex(), how)
    assert seen == {"q", "side", "tie", "division"}
