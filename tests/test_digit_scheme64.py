"""The seven-digit contraction of the FP64 plans' tensor-core Legendre kernels,
restated in integers (the arithmetic of cunusht_gb300/csrc/rec64.cuh and
legendre_tc64.cu, independent of the GPU): X = trunc(v 2^55) for |v| < 1 as
balanced base-256 digits, digit products of weight i + j <= 6 summed over a
128-l window in FP32, combined in 64-bit integers."""
import numpy as np
import pytest

BIAS = 0x0080808080808080


def fix55_biased(v, eb=0):
    """Bit-for-bit the device function (sign, shift and bias on integers)."""
    u = int(np.float64(v).view(np.uint64))
    e, neg = (u >> 52) & 0x7FF, u >> 63
    n = min((1030 + eb - e) & 0xFFFFFFFF, 63)
    big = ((u & 0xFFFFFFFFFFFFF) | (1 << 52)) << 10
    return ((-(big >> n) if neg else big >> n) + BIAS) & 0xFFFFFFFFFFFFFFFF


def digits(word):
    return [((word >> 48) & 0xFFFF) - 128] + [((word >> (8 * (6 - k))) & 0xFF) - 128 for k in range(1, 7)]


@pytest.mark.parametrize("v", [0.0, 1.0 - 2.0 ** -53, -1.0 + 2.0 ** -53, 0.5, -0.5, 2.0 ** -55, -2.0 ** -55, 2.0 ** -56,
                               1 / 3, -1 / 3, 255 / 256, 1e-10, -1e-300, 2.0 ** -1074])
def test_digits_are_the_truncated_value(v):
    d = digits(fix55_biased(v))
    assert all(-128 <= x <= 128 for x in d)
    assert sum(x * 256 ** (6 - k) for k, x in enumerate(d)) == int(np.trunc(np.longdouble(v) * 2 ** 55))


def test_digits_random_and_shifted():
    rng = np.random.default_rng(0)
    for v in rng.uniform(-1, 1, 2000) * 2.0 ** -rng.integers(0, 70, 2000):
        for eb in (0, 3, -2):
            if abs(v) >= 2.0 ** eb:
                continue
            d = digits(fix55_biased(v, eb))
            assert sum(x * 256 ** (6 - k) for k, x in enumerate(d)) == int(np.trunc(np.longdouble(v) * 2.0 ** (55 - eb)))


def test_window_sums_are_exact_in_fp32():
    """The largest sum of one weight: 7 digit pairs of 128 x 128 over 128 l."""
    assert 7 * 128 * 128 * 128 < 2 ** 24


def test_contraction_error():
    """Truncation of both factors and the dropped weights: below 2^-52 of the bounds per term."""
    rng = np.random.default_rng(1)
    a, b = rng.uniform(-1, 1, (2, 128))
    da, db = ([digits(fix55_biased(x)) for x in y] for y in (a, b))
    total = 0
    for g in range(7):
        s = sum(da[l][i] * db[l][g - i] for l in range(128) for i in range(g + 1))
        assert abs(s) < 2 ** 24
        total += s * 256 ** (6 - g)
    want = sum(int(x * 2 ** 60) * int(y * 2 ** 60) for x, y in zip(a, b)) / 2 ** 120
    assert abs(total / 2 ** 62 - want) < 128 * 2.0 ** -52
