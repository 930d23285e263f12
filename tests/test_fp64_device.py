"""The arithmetic of csrc/fp64.cuh on the GPU against CUDA's own product, quotient and comparisons, bit for bit:
random values of ordinary and extreme exponents, short mantissas (ties, exact results, carries), and every
pair of the ends of the ranges, zeros, subnormals, infinities and NaN."""
import ctypes as C

import numpy as np
import pytest

import device

OPS = ["mul", "mul_float", "div", "rcp", "div_stored", "div_two", "half", "quarter", "negative", "nonzero", "upwind",
       "positive"]
INF, NAN = float("inf"), float("nan")
EDGES = [0.0, 5e-324, 2.0 ** -1074 * 12345, 2.0 ** -1022, 2.0 ** -1021, 2.0 ** -970, 2.0 ** -511, 2.0 ** -510,
         np.nextafter(2.0 ** -510, 1), 2.0 ** -149, 2.0 ** -127, 2.0 ** -126, 2.0 ** -101, 2.0 ** -100, 1e-30, 1 / 3, 1.0,
         np.nextafter(1.0, 2), 1.5, 3.0, 1e5, 2.0 ** 99, np.nextafter(2.0 ** 100, 0), 2.0 ** 100, 2.0 ** 127, 2.0 ** 128,
         np.nextafter(2.0 ** 512, 0), 2.0 ** 512, 2.0 ** 1022, 1.7e308, INF, NAN]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return device.library("device_fp64.cu", "kernels_fp64.cu", tmp_path_factory.mktemp("fp64"))


def apply(lib, op, a, b, c=None):
    c = np.ones_like(a) if c is None else c
    a, b, c = (np.ascontiguousarray(v, np.float64) for v in (a, b, c))
    r, s = np.zeros_like(a), np.zeros_like(a)
    p = lambda v: v.ctypes.data_as(C.c_void_p)
    assert lib.fp64_op(OPS.index(op), C.c_longlong(a.size), p(a), p(b), p(c), p(r), p(s)) == 0
    return r, s


def same(r, s, zero_sign=True):
    """equal bits (NaN equals NaN)"""
    eq = (r.view(np.uint64) == s.view(np.uint64)) | (np.isnan(r) & np.isnan(s))
    return eq if zero_sign else eq | ((r == 0.0) & (s == 0.0))


def values(kind, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = {"ordinary": (-60, 60), "wide": (-480, 480), "short": (-20, 20)}[kind]
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    if kind == "short":
        m &= np.uint64(0xFFFFFFC000000) | np.uint64(rng.integers(0, 1 << 52))
    e = rng.integers(1023 + lo, 1023 + hi, n).astype(np.uint64)
    s = rng.integers(0, 2, n).astype(np.uint64)
    return ((s << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)


def edge_pairs():
    v = np.array(EDGES + [-x for x in EDGES])
    a, b = np.meshgrid(v, v)
    return a.ravel(), b.ravel()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["ordinary", "wide", "short"])
@pytest.mark.parametrize("op", ["mul", "mul_float", "div", "rcp", "div_stored", "half", "quarter"])
def test_random_values(op, kind, lib):
    n = 1 << 20
    a, b = values(kind, n, 1), values(kind, n, 2)
    if op == "mul_float":
        a = np.clip(a, -3e38, 3e38)
    if op in ("div", "div_stored") and kind == "wide":
        b = values("ordinary", n, 3)  # the divisors' range; quotients stay normal
    r, s = apply(lib, op, a, b)
    bad = ~same(r, s)
    assert not bad.any(), (a[bad][:3], b[bad][:3], r[bad][:3], s[bad][:3])


@pytest.mark.gpu
def test_quotient_by_a_product_of_two(lib):
    """The reciprocal is a product of a stored one and of rcp_near's, the divisor a rounded product."""
    n = 1 << 20
    a, b, c = (values("ordinary", n, k) for k in (4, 5, 6))
    r, s = apply(lib, "div_two", a, b, np.abs(c) ** 0.5)
    bad = ~same(r, s)
    assert not bad.any(), (a[bad][:3], b[bad][:3], c[bad][:3])


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["mul", "mul_float", "half", "quarter"])
def test_edges_of_products(op, lib):
    a, b = edge_pairs()
    r, s = apply(lib, op, a, b)
    bad = ~same(r, s)
    assert not bad.any(), list(zip(a[bad], b[bad], r[bad], s[bad]))[:5]


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["div", "rcp", "div_stored"])
def test_edges_of_quotients(op, lib):
    """As fp64.cuh states them: not the sign of a zero quotient; a quotient of a dividend below 2^-960 may be
    off by the smallest subnormal, or by a unit where it is normal; div_rn's divisors are within 2^-100..2^99
    or 0, infinite, NaN."""
    a, b = edge_pairs()
    if op == "div_stored":
        with np.errstate(all="ignore"):
            m = np.abs(b)
            keep = ~((m > 0) & (m < 2.0 ** -100)) & ~((m >= 2.0 ** 100) & np.isfinite(m))
        a, b = a[keep], b[keep]
    r, s = apply(lib, op, a, b)
    ok = same(r, s, zero_sign=op == "rcp")
    if op != "rcp":
        tiny = np.abs(a) < 2.0 ** -960
        with np.errstate(all="ignore"):
            ok |= tiny & (np.abs(r - s) <= np.maximum(np.spacing(np.abs(s)), 5e-324))
            # a quotient below the normal range
            ok |= (np.abs(s) < 2.0 ** -1022) & (np.abs(r - s) <= 5e-324)
    assert ok.all(), list(zip(a[~ok], b[~ok], r[~ok], s[~ok]))[:5]


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["negative", "nonzero", "upwind", "positive"])
def test_comparisons_by_the_bits(op, lib):
    """As fp64.cuh states them: -0 counts as negative, a positive NaN as upwind and positive."""
    a, _ = edge_pairs()
    a = np.concatenate([a, values("ordinary", 4096, 8)])
    r, s = apply(lib, op, a, a)
    nan, neg0 = np.isnan(a), (a == 0.0) & np.signbit(a)
    if op == "negative":
        s[neg0] = 1.0
    if op == "upwind":
        s[nan] = ~np.signbit(a[nan])
    if op == "positive":
        s[nan] = ~np.signbit(a[nan])
    np.testing.assert_array_equal(r, s)
