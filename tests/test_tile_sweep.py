"""The tiled vertical solve's forward and back substitution keep their FP64 right-hand sides in FP64: with FP32
coefficients they give what the same elimination gives with every row divided in FP64.

The bar: a multiplier is good to 2^-45, a sum of products to 2^-53; with factors of at most 1 (diagonally
dominant rows) n rows down and n back add at most 2*n of these, 2*128*2^-45 = 2^-37 of the largest
solution.  (A multiplier rounded to FP32 is off by up to 2^-24.)
"""
import ctypes as C

import numpy as np
import pytest

import device


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return device.library("device_sweep.cu", "split.cu", tmp_path_factory.mktemp("sweep"))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n, cols", [(2, 1), (23, 33), (79, 96), (127, 64)])
def test_substitutions_keep_fp64(n, cols, dtype, lib):
    rng = np.random.default_rng(n)
    c, e = (rng.uniform(0.5, 1.0, (n, cols)) for _ in range(2))
    up = np.vstack([np.zeros((1, cols)), c[:-1]])
    d = -1.01 * (up + e)
    c, e, d = (np.ascontiguousarray(1e-7 * a, dtype) for a in (c, e, d))  # the vertical solve's magnitude
    rhs = np.ascontiguousarray(rng.normal(size=(n, cols)))
    tile, plain = np.zeros((n, cols)), np.zeros((n, cols))
    f = lib.sweeps_f32 if dtype == np.float32 else lib.sweeps_f64
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    assert f(n, cols, p(d), p(c), p(e), p(rhs), p(tile), p(plain)) == 0
    assert np.isfinite(plain).all() and np.abs(plain).min() > 0.0
    err = np.abs(tile - plain).max(0) / np.abs(plain).max(0)
    assert err.max() <= 2.0 ** -37, err.max()
