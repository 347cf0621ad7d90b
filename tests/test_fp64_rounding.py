"""The FP64 walk's root and quotient (walk_ops.cuh, fp64_contrib) where they are hardest to
round: square roots and quotients within 2^-44 units in the last place of the
midpoint of two doubles.  On the CPU the function is restated operation by
operation, with its float approximation up to two units off; on the GPU it runs
itself (tests/device/probe.cu).  Both must give the correctly rounded results."""
import math
import struct
from fractions import Fraction

import numpy as np
import pytest

from device_probe import probe  # noqa: F401

# r (53 bits) and m (24 bits) with m 2^t = M r + c for an odd 54-bit M and c = +-1, +-3: m / r
# next to the midpoint M, found by factoring m 2^t - c.  Without near_half the function
# misses each of these with one of the approximations below at least.
QUOTIENTS = [
    (0x157a028343fd73, 0x97a4e9), (0x15948070112b8d, 0xb4521d), (0x16b1f1f66cb7e7, 0x83059d),
    (0x17695ffe461265, 0xbb9ac3), (0x17c494d0ca7181, 0xa88073), (0x186bb0f5c42831, 0xd7494f),
    (0x186e384e8db8e7, 0xbc9ae3), (0x18bfde01577bd1, 0x8a9643), (0x191581fc5aca89, 0xf8c3e9),
    (0x192a9fbcac6129, 0xe7f52d), (0x1964677461a403, 0xc85b73), (0x196bd88a00cd03, 0x8490a9),
    (0x19e1c1f7e89aa3, 0xaea499), (0x19fb377856e6c7, 0xc6cc05), (0x1a2c27528112d9, 0xbbda0d),
    (0x1a4e84c61d54d5, 0xb9ac15), (0x1a802e49257d9f, 0xe4291b), (0x1a8dbcc69c6403, 0xcc2209),
    (0x1acd3be601e53b, 0x85e77d), (0x1b1eb408076631, 0xa9faf1), (0x1b4128a7d82ced, 0x9c578f),
    (0x1ba470ca561a6b, 0xc01fe5), (0x1c06f9441d8bfb, 0xfd01f5), (0x1c4b70b6825291, 0xed1083),
    (0x1c972decb528b9, 0xaeefa3), (0x1c9bfdf0b0b507, 0xec958b), (0x1c9dc434ad30e5, 0xcf17e7),
    (0x1cabc01066469f, 0xa2e2c7), (0x1cd1216176d8d5, 0xb9bd3b), (0x1cf29fed773ead, 0x8bbc97),
    (0x1cf3a57cfb7281, 0xa53677), (0x1d06cd2f3da611, 0xf28a15), (0x1d34cce011255f, 0x8c18cd),
    (0x1dc2346b0dc517, 0xd49de5), (0x1ddfd3465accdb, 0xf69975), (0x1e0b172ebb20d5, 0x8490a9),
    (0x1e15c771a5be69, 0xcd911b), (0x1e1b376c4ff79f, 0xabb8f3), (0x1e530882c16155, 0xee27af),
    (0x1e7c73ab987a8b, 0xbbf495), (0x1e975cf25f286f, 0xe3db01), (0x1ea3d1bb064d3b, 0xfd6521),
    (0x1ec82acd6e67b1, 0xfd2187), (0x1eda90a42228a9, 0xf8c3e9), (0x1eeedfbfcbff7f, 0xd8c7e7),
    (0x1ef3475c7117e3, 0xb76061), (0x1f1dc50bfcbc8b, 0xf6361f), (0x1f213d59c0bda5, 0xfcaf8b),
    (0x1f413bf35310a3, 0x8ead67), (0x1f517905056eed, 0xd17443), (0x1f5f9fb92b7d7f, 0xc42239),
    (0x1f6904e6b9c563, 0xdb8e8f), (0x1f78526389bb99, 0xe55a8b), (0x1f920f32c03ed7, 0x8a5b0d),
    (0x1f9f4e77704379, 0xc1cb71), (0x1fd61d19789653, 0xea4517), (0x1fdda0c8491ce1, 0xdc0f1d),
    (0x1ff8aff3168679, 0x96e0fd),
]


def roots(most=400):
    """Doubles r2 with r2 2^k = M^2 + c for an odd 54-bit M and |c| <= most: M by Hensel's
    lifting of a square root of -c modulo a power of two."""
    out = []
    for c in range(-most - most % 8 - 1, most, 8):  # -c = 1 (mod 8): the odd squares
        for b in (54, 55):
            x = 1
            for k in range(3, b):
                x += (x * x + c) % (1 << (k + 1)) and 1 << (k - 1)
            for root in {s * x + h for s in (1, -1) for h in (0, 1 << (b - 1))}:
                m = root % (1 << b)
                while m < 1 << 54:
                    v = m * m + c
                    if m >= 1 << 53 and v % (1 << b) == 0 and v >> b < 1 << 53:
                        out.append(math.ldexp(v >> b, b - 106))
                    m += 1 << b
    return sorted(set(out))


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def near_half(x, y):
    return ((bits(x) - bits(y) + 64) & ((1 << 52) - 1)) <= 128


def root_and_quotient(r2, m, y):
    """fp64_contrib's, or None where it leaves them to the library operations."""
    g, k = r2 * y, 0.5 * y
    e = fma(-g, k, 0.5)
    g, k = fma(g, e, g), fma(k, e, k)
    e = fma(-g, k, 0.5)
    g, k = fma(g, e, g), fma(k, e, k)
    rem = fma(-g, g, r2)
    r = fma(rem, k, g)
    inv = 2.0 * k
    q = m * inv
    q = fma(fma(-q, r, m), inv, q)
    qrem = fma(-q, r, m)
    if near_half(rem, g) or near_half(qrem, r):
        return None
    return r, fma(qrem, inv, q)


def cases():
    near = [(math.ldexp(r, -52) ** 2, math.ldexp(m, -22)) for r, m in QUOTIENTS]
    return near + [(r2, m) for r2 in roots() for m in (1.0, 0.7)]


def test_the_cases_are_hard():
    for r, m in QUOTIENTS:
        q = Fraction(m, r)
        q *= 2 ** (54 - (q.numerator.bit_length() - q.denominator.bit_length()))
        q = q if q < 2 ** 54 else q / 2
        odd = 2 * (q // 2) + 1  # the midpoint in units of half a last place
        assert 0 < abs(q - odd) <= Fraction(8, 1 << 52)
    assert len(roots()) > 100
    for r2 in roots():
        n, d = r2.as_integer_ratio()
        k = 107 - n.bit_length()
        k += (k + d.bit_length() - 1) % 2  # r2 as a square of a 54-bit number, nearly
        v = n << k
        odd = math.isqrt(v)
        odd += odd % 2 == 0
        assert abs(v - odd * odd) <= 408


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])
def test_root_and_quotient_next_to_midpoints(ulps):
    for r2, m in cases():
        m = float(np.float32(m))
        y0 = np.float32(1.0 / math.sqrt(float(np.float32(r2))))
        y = float((y0.view(np.uint32) + np.uint32(ulps & 0xFFFFFFFF)).view(np.float32))
        got = root_and_quotient(r2, m, y)
        r = math.sqrt(r2)
        assert got is None or got == (r, m / r), (r2.hex(), m.hex())


def test_ordinary_inputs_do_not_leave_it():
    rng = np.random.default_rng(5)
    left = 0
    for _ in range(2000):
        s = (rng.uniform(-1, 1, 3) * 10.0 ** rng.uniform(-4, 2)).astype(np.float32)
        r2 = float(s[0]) ** 2 + float(s[1]) ** 2 + float(s[2]) ** 2
        m = float(np.float32(math.exp(rng.uniform(-12, 8))))
        left += root_and_quotient(r2, m, float(np.float32(1.0 / math.sqrt(r2)))) is None
    assert left == 0


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0, 17, -40])
@pytest.mark.parametrize("softening", [2.0 ** -30, 2.0 ** 30])
def test_device_function(probe, scale, softening):
    """-m / r and, inside the softening length, the spline, bit for bit."""
    rng = np.random.default_rng(7)
    near = cases()
    s = rng.uniform(-1, 1, (1 << 18, 3)).astype(np.float32).astype(np.float64)
    s *= 10.0 ** rng.integers(-4, 3, (len(s), 1))
    r2 = np.concatenate([[c[0] for c in near], (s * s).sum(1)]) * 4.0 ** scale
    m = np.concatenate([[c[1] for c in near],
                        np.exp(rng.uniform(-12, 8, len(s)))]).astype(np.float32)
    got, want = probe.call("probe_fp64_contrib", r2, np.float64, m, softening * 2.0 ** scale)
    probe.same_bits(got, want, r2, m)
    if softening < 1e-6:  # the library operations are the correctly rounded ones
        assert np.array_equal(want, -(m.astype(np.float64) / np.sqrt(r2)))
