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
