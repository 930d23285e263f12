"""The integer product and the reciprocal of fp64.cuh, restated in exact integer and rational
arithmetic on the CPU: mul_int rounds the product of two doubles to nearest even; rcp_near's Halley
step, from a reciprocal good to 2^-22, is within two units of the last place of 1/b, and one
quotient, remainder and correction then give the rounded quotient (div_rn)."""
import struct
from fractions import Fraction

import numpy as np
import pytest

M32 = (1 << 32) - 1


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def of_bits(u):
    return struct.unpack("<d", struct.pack("<Q", u))[0]


def mul_int(x, y):
    """mul_int of csrc/fp64.cuh, word by word; None where it takes the hardware's product."""
    xh, xl, yh, yl = bits(x) >> 32, bits(x) & M32, bits(y) >> 32, bits(y) & M32
    xe, ye = xh & 0x7FF00000, yh & 0x7FF00000
    if max((xe - (513 << 20)) & M32, (ye - (513 << 20)) & M32) >= (1022 << 20):
        return None

    def shf(lo, hi, s):
        return (((hi << 32) | lo) << s >> 32) & M32
    ah, al = (shf(xl, xh, 1) & 0x1FFFFF) | 0x200000, (xl << 1) & M32
    bh, bl = shf(yl, yh, 11) | 0x80000000, (yl << 11) & M32
    p00 = al * bl
    p01 = al * bh + (p00 >> 32)
    p10 = ah * bl + (p01 & M32)
    up = ah * bh + (p01 >> 32) + (p10 >> 32)
    assert max(p00, p01, p10, up) < 1 << 64
    hh, hl, mid = up >> 32, up & M32, p10 & M32
    big = hh >> 21
    sh = 1 - big
    hh, hl = shf(hl, hh, sh), shf(mid, hl, sh)
    t = ((hl >> 1) & 1) | (1 if (((mid << sh) & M32) | (p00 & M32)) else 0)
    r = (((hh << 32) | hl) + t) >> 1
    e = (xe + ye - 0x3FF00000 - 0x00100000 + (big << 20)) & M32
    return of_bits(((((r >> 32) + e) & M32) ^ ((xh ^ yh) & 0x80000000)) << 32 | (r & M32))


def pairs(kind, n=20000):
    rng = np.random.default_rng(7)
    ex = {"ordinary": (983, 1063), "window": (513, 1535)}.get(kind, (1000, 1046))
    u = rng.integers(0, 1 << 52, (n, 2), dtype=np.uint64)
    if kind == "ties":  # short mantissas: exact products, halves and carries
        u &= np.uint64(0xFFFFFFFFC000000) | np.uint64(1 << 26)
    if kind == "ones":
        u |= np.uint64((1 << 52) - (1 << 20))
    e = rng.integers(*ex, (n, 2)).astype(np.uint64)
    s = rng.integers(0, 2, (n, 2)).astype(np.uint64)
    return ((s << np.uint64(63)) | (e << np.uint64(52)) | u).view(np.float64)


@pytest.mark.parametrize("kind", ["ordinary", "window", "ties", "ones"])
def test_integer_product_is_the_rounded_product(kind):
    for x, y in pairs(kind):
        assert bits(mul_int(x, y)) == bits(float(x) * float(y)), (x, y)


def test_integer_product_leaves_the_ends_of_the_range_to_the_hardware():
    for x, y in [(2.0 ** -511, 1.0), (1.0, 2.0 ** 512), (0.0, 1.0), (float("inf"), 1.0), (1.0, float("nan")), (5e-324, 1.0)]:
        assert mul_int(x, y) is None
    assert mul_int(2.0 ** -510, 2.0 ** -510) == 2.0 ** -1020 and mul_int(-2.0 ** 511, 2.0 ** 511) == -2.0 ** 1022


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def test_quotient_is_the_rounded_quotient():
    rng = np.random.default_rng(3)
    for x, y in pairs("ordinary", 4000):
        x, y = float(x), float(y)
        y0 = float(np.float32(1.0) / np.float32(y)) * (1.0 + rng.uniform(-1.0, 1.0) * 2.0 ** -23)
        e = fma(-y, y0, 1.0)
        r = fma(y0, fma(e, e, e), y0)
        assert abs(Fraction(r) * Fraction(y) - 1) < Fraction(1, 1 << 51)
        q = x * r
        assert fma(fma(-y, q, x), r, q) == x / y
        assert fma(fma(-y, r, 1.0), r, r) == 1.0 / y


def mul_int_single(x, y):
    """mul_int of csrc/fp64.cuh with a single-precision factor x; None where it takes the hardware's product."""
    xu = struct.unpack("<I", struct.pack("<f", x))[0]
    yh, yl = bits(y) >> 32, bits(y) & M32
    xe, ye = xu & 0x7F800000, yh & 0x7FF00000
    if (xe - (1 << 23)) & M32 >= 254 << 23 or (ye - (513 << 20)) & M32 >= 1022 << 20:
        return None
    a = (xu << 8) & M32 | 0x80000000
    bh, bl = (((yh << 32 | yl) << 1) >> 32 & 0x1FFFFF) | 0x200000, (yl << 1) & M32
    low = a * bl
    up = a * bh + (low >> 32)
    assert max(low, up) < 1 << 64
    hh, hl, mid = up >> 32, up & M32, low & M32
    big = hh >> 21
    assert big in (0, 1)
    sh = 1 - big
    hh, hl = (((hh << 32 | hl) << sh) >> 32) & M32, (((hl << 32 | mid) << sh) >> 32) & M32
    t = (hl >> 1 & 1) | (1 if (mid << sh) & M32 else 0)
    r = (((hh << 32 | hl) + t) & ((1 << 64) - 1)) >> 1
    e = (xe >> 3) + (896 << 20) + ye - 0x3FF00000 - 0x00100000 + (big << 20)
    return of_bits((((((r >> 32) + e) & M32) ^ ((xu >> 31 ^ yh >> 31) << 31)) << 32) | (r & M32))


@pytest.mark.parametrize("kind", ["ordinary", "window", "ties", "ones"])
def test_integer_product_with_a_single_precision_factor(kind):
    for x, y in pairs(kind):
        x = float(np.float32(x)) if 2.0 ** -126 <= abs(float(x)) < 2.0 ** 127 else 1.0 + float(x) % 1.0
        x = float(np.float32(x))
        assert bits(mul_int_single(x, float(y))) == bits(x * float(y)), (x, y)
    for x, y in [(0.0, 1.0), (2.0 ** -127, 1.0), (float("inf"), 1.0), (float("nan"), 1.0), (1.0, 2.0 ** 512), (1.0, 0.0)]:
        assert mul_int_single(x, y) is None
