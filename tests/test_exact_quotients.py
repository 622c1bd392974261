"""The corrected quotients of the shading and traversal kernels (byte_over_255 and over_pi in
device_math.cuh, quotient_f64 in traverse.cuh) give the IEEE quotient: the same operations restated
here, with rounding of exact values."""
import random
from fractions import Fraction as F

import numpy as np
import pytest


def rounded(x, bits):
    """The nearest `bits`-bit binary fraction, ties to even."""
    if x == 0:
        return F(0)
    sign, x = (-1 if x < 0 else 1), abs(x)
    e = x.numerator.bit_length() - x.denominator.bit_length()
    if x < F(2) ** e:
        e -= 1
    m = x / F(2) ** (e - bits + 1)
    n = m.numerator // m.denominator
    r = m - n
    if r > F(1, 2) or (r == F(1, 2) and n & 1):
        n += 1
    return sign * n * F(2) ** (e - bits + 1)


def test_byte_over_255():
    rc = rounded(F(1, 255), 24)
    for b in range(256):
        q = rounded(b * rc, 24)
        r = rounded(b - q * 255, 24)
        assert rounded(q + r * rc, 24) == rounded(F(b, 255), 24), b


@pytest.mark.parametrize("exponent", [0, -1, -30])
def test_over_pi_for_every_mantissa(exponent):
    pi = np.float32(3.14159265358979323846)
    rc = np.float32(1.0 / np.float64(pi))
    x = (np.arange(1 << 23, dtype=np.uint32) | np.uint32((127 + exponent) << 23)).view(np.float32)
    want = (x.astype(np.float64) / np.float64(pi)).astype(np.float32)  # 53 >= 2 * 24 + 2 bits: rounds once
    q = x * rc
    # x - q pi and q + r rc exactly in 64 mantissa bits, then rounded
    r = (x.astype(np.longdouble) - q.astype(np.longdouble) * np.longdouble(pi)).astype(np.float32)
    got = (q.astype(np.longdouble) + r.astype(np.longdouble) * np.longdouble(rc)).astype(np.float32)
    assert np.array_equal(got, want)


def test_quotient_f64_of_f32_operands():
    rng = random.Random(5)
    edge = [1 << 23, (1 << 23) + 1, (1 << 24) - 1, (1 << 24) - 2, 0xAAAAAB, 0xD55555]
    for _ in range(20000):
        a = F(rng.choice(edge) if rng.random() < 0.3 else rng.randrange(1 << 23, 1 << 24)) * F(2) ** rng.randint(-120, 0)
        b = F(rng.choice(edge) if rng.random() < 0.3 else rng.randrange(1 << 23, 1 << 24))
        y = rounded(1 / b, 53)
        q = rounded(a * y, 53)
        q = rounded(q + rounded(a - b * q, 53) * y, 53)
        assert rounded(q + rounded(a - b * q, 53) * y, 53) == rounded(a / b, 53)
