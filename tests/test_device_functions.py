"""The device code's scalar functions themselves (tests/device/probe.cu includes the
library's headers) against the operations they stand for, bit for bit: values
of every exponent, the special ones, and the inputs next to a rounding boundary."""
import numpy as np
import pytest

from device_probe import probe  # noqa: F401

pytestmark = pytest.mark.gpu


def floats(rng, n):
    """Every exponent and sign, zeros, subnormals, infinities and NaNs."""
    special = np.array([0, 0x80000000, 1, 0x80000001, 0x7FFFFF, 0x800000, 0x7F7FFFFF, 0x7F800000,
                        0xFF800000, 0x7F800001, 0xFF800001, 0x7FC00000, 0xFFC00000, 0x7FFFFFFF,
                        0xFFFFFFFF, 0x7FA12345, 0xFFD54321], np.uint32)
    return np.concatenate([special, rng.integers(0, 1 << 32, n, np.uint64).astype(np.uint32)]) \
        .view(np.float32)


def doubles(rng, n):
    special = np.array([0, 1 << 63, 1, (1 << 63) | 1, 0x7FF0000000000000, 0xFFF0000000000000,
                        0x7FF0000000000001, 0xFFF0000000000001, 0x7FF8000000000000,
                        0xFFF8000000000000, 0x7FFFFFFFFFFFFFFF, 0xFFFFFFFFFFFFFFFF,
                        0x7FF4000012345678, 0xFFF4000012345678], np.uint64)
    # exponents around the floats' range (2^-160 .. 2^140), mantissas on and next to ties
    ex = rng.integers(1023 - 160, 1023 + 140, n).astype(np.uint64)
    top = rng.integers(0, 1 << 23, n).astype(np.uint64) << np.uint64(29)
    low = rng.choice(np.array([0, 1, (1 << 28) - 1, 1 << 28, (1 << 28) + 1, (1 << 29) - 1],
                              np.uint64), n)
    sub = rng.integers(0, 1 << 52, n).astype(np.uint64)  # subnormal results: ties anywhere
    sub &= ~((np.uint64(1) << rng.integers(0, 53, n).astype(np.uint64)) - np.uint64(1))
    sign = rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63)
    mant = np.where(ex < np.uint64(1023 - 126), sub, top | low)
    return np.concatenate([special, sign | (ex << np.uint64(52)) | mant,
                           rng.integers(0, 1 << 64, n, np.uint64)]).view(np.float64)


def test_float_to_double_is_the_conversion(probe):
    x = floats(np.random.default_rng(1), 1 << 20)
    got, want = probe.call("probe_f2d", x, np.float64)
    signalling = np.isnan(x) & (x.view(np.uint32) & 0x400000 == 0)
    got.view(np.uint64)[signalling] |= 1 << 51  # quieted by the next operation
    probe.same_bits(got, want, x.view(np.uint32))


def test_double_to_float_is_the_conversion(probe):
    x = doubles(np.random.default_rng(2), 1 << 20)
    got, want = probe.call("probe_d2f", x, np.float32)
    probe.same_bits(got, want, x.view(np.uint64))


@pytest.mark.parametrize("a", [1.0, 0.5, 0.3, 0.7123457, 0.99999994, 1.0000001, 3.0e-3, 12.5])
def test_over_the_scale_factor_is_the_division(probe, a):
    rng = np.random.default_rng(int(a * 1e6))
    a = np.float32(a)
    n = 1 << 19
    x = np.concatenate([doubles(rng, n), -np.exp(rng.uniform(-60, 60, n)),
                        # next to and on multiples of the divisor
                        (rng.uniform(1, 2, n) * float(a)) * 2.0 ** rng.integers(-40, 40, n)])
    x = x[~np.isnan(x)]
    got, want = probe.call("probe_over_scale", x, np.float64, a)
    probe.same_bits(got, want, x)


def test_centre_of_mass_quotient_is_the_rounded_division(probe):
    """float(c / m): moments of two to eight float masses, quotients next to and on the
    midpoints of two floats, and every exponent."""
    rng = np.random.default_rng(11)
    n = 1 << 19
    w = np.exp(rng.uniform(-8, 8, (n, 8))).astype(np.float32).astype(np.float64)
    w *= np.arange(8) < rng.integers(2, 9, (n, 1))
    w[: n // 2] = (w[: n // 2] > 0) * w[: n // 2, :1]  # equal masses: ties
    x = rng.normal(0, 1, (n, 8)).astype(np.float32).astype(np.float64)
    c, m = (w * x).sum(1), w.sum(1)
    mid = (rng.integers(1 << 24, 1 << 25, n) | 1) * 2.0 ** rng.integers(-60, 20, n)
    mm = np.exp(rng.uniform(-20, 20, n))
    near = mid * mm * (1 + rng.integers(-3, 4, n) * 2.0 ** -52)
    wild = rng.integers(0, 1 << 64, (2, n), np.uint64).view(np.float64)
    c = np.concatenate([c, near, -near, mid * 3, wild[0]])
    m = np.concatenate([m, mm, mm, np.full(n, 3.0), wild[1]])
    got, want = probe.call("probe_quot_float", c, np.float32, m)
    probe.same_bits(got, want, c, m)


@pytest.mark.parametrize("kind", ["masses", "positive", "signed", "wide", "ties", "borders", "inf",
                                  "nan", "zero", "tiny"])
@pytest.mark.parametrize("K", [1, 7, 18])
def test_sums_of_many_chunks_are_the_loop(probe, kind, K):
    """Every column of every subhalo of at least 64 chunks, bit for bit; shorter ones keep
    their chunks' sums."""
    import ctypes as C

    from test_sum_in_order import _terms
    rng = np.random.default_rng(K)
    chunks = [63, 64, 65, 1999, 96, 40, 127]
    base = np.concatenate([[0], np.cumsum(chunks)]).astype(np.int32)
    order = np.argsort(-np.array(chunks), kind="stable").astype(np.int32)
    sums = np.zeros((base[-1], 24))
    for s, n in enumerate(chunks):
        for k in range(24):
            sums[base[s]:base[s + 1], k] = _terms(kind, n, rng)
    before = sums.copy()
    loop = np.zeros((len(order), K))
    with np.errstate(all="ignore"):
        assert probe.lib.probe_fold(*(C.c_void_p(a.ctypes.data) for a in (sums, base, order)),
                                    len(chunks), len(order), K, C.c_void_p(loop.ctypes.data)) == 0
    for j, s in enumerate(order):
        if chunks[s] >= 64:
            got, want = sums[base[s], :K].copy(), loop[j]
            nan = np.isnan(want)
            assert np.array_equal(np.isnan(got), nan)
            assert np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64)), (s, K)
            before[base[s], :K] = got
    assert np.array_equal(sums.view(np.uint64), before.view(np.uint64))  # and nothing else
