"""float <-> double from the IEEE-754 fields (device_common.cuh, f2d and d2f),
restated on integers: every result must have the bits of the plain conversion,
at the edges of the formats (zeros, subnormals, ties, carries, overflow,
infinities) and on random bit patterns."""
import numpy as np
import pytest


def f2d(x):
    u = x.view(np.uint32).astype(np.uint64)
    e = (u >> 23) & 0xFF
    with np.errstate(invalid="ignore"):
        y = (x * np.float32(2.0) ** 64).view(np.uint32).astype(np.uint64)
    sub = e == 0
    u2 = np.where(sub, y, u)
    bias = np.where(sub, np.where(u2 & 0x7FFFFFFF, 896 - 64, 0), 896)
    bias = np.where(e == 0xFF, 0x7FF - 0xFF, bias).astype(np.uint64)
    hi = (u & 0x80000000) | ((((u2 >> 23) & 0xFF) + bias) << 20) | ((u2 & 0x7FFFFF) >> 3)
    return (hi << 32) | ((u2 << 29) & 0xFFFFFFFF)


def d2f(x):
    b = x.view(np.uint64)
    e = ((b >> 52) & 0x7FF).astype(np.int64) - 896
    mant = b & 0xFFFFFFFFFFFFF
    up = ((b & 0x1FFFFFFF) + ((mant >> 29) & 1)) > (1 << 28)
    bits = (e << 23) + (mant >> 29).astype(np.int64) + up
    s = np.clip(30 - e, 1, 63).astype(np.uint64)
    m = mant | (1 << 52)
    q, rem, half = m >> s, m & ((np.uint64(1) << s) - np.uint64(1)), np.uint64(1) << (s - np.uint64(1))
    low = np.where(s > 53, 0, q.astype(np.int64) + ((rem + (q & 1)) > half))
    inf = np.where((e == 0x7FF - 896) & (mant != 0), 0x7FC00000, 0x7F800000)
    bits = np.where(e <= 0, low, np.where((e >= 255) | (bits >= 0x7F800000), inf, bits))
    return (bits.astype(np.uint64) | ((b >> 63) << 31)).astype(np.uint32)


@pytest.mark.parametrize("kind", ["edges", "random"])
def test_conversions(kind):
    rng = np.random.default_rng(7)
    if kind == "edges":
        f = np.array([0, 1, 2, 0x7FFFFF, 0x800000, 0x800001, 0x7F7FFFFF, 0x7F800000], np.uint32)
        f = np.concatenate([f, f | np.uint32(0x80000000)])
        d = np.concatenate([[0], (np.uint64(1) << np.arange(53, dtype=np.uint64)) - np.uint64(1)])
        d = np.concatenate([(d.astype(np.uint64) & ((1 << 52) - 1)) | (np.uint64(k) << 52)
                            for k in (0, 870, 871, 872, 873, 895, 896, 897, 1023, 1150, 1151, 2046)])
        ties = (np.arange(64, dtype=np.uint64) << 29) | (1 << 28)
        d = np.concatenate([d, ties | (np.uint64(1023) << 52), ties | (np.uint64(880) << 52),
                            np.array([0x7FF << 52], np.uint64)])
        d = np.concatenate([d, d | np.uint64(1 << 63)])
    else:
        f = rng.integers(0, 1 << 32, 200000, np.uint64).astype(np.uint32)
        d = rng.integers(0, 1 << 64, 200000, np.uint64)
        d[::2] = (d[::2] & ~np.uint64(0x7FF << 52)) | (
            rng.integers(860, 1160, len(d[::2]), np.uint64) << np.uint64(52))
        d[::3] = (d[::3] & ~np.uint64(0x1FFFFFFF)) | np.uint64(1 << 28)
    f, d = f.view(np.float32), d.view(np.float64)
    f, d = f[~np.isnan(f)], d[~np.isnan(d)]
    assert np.array_equal(f2d(f), f.astype(np.float64).view(np.uint64))
    with np.errstate(over="ignore"):
        assert np.array_equal(d2f(d), d.astype(np.float32).view(np.uint32))
