"""Square roots of the diagonal blocks' pivots and their reciprocals against CUDA's sqrt and reciprocal, bit for bit: the
iteration's error before its last rounding is below 2^-86, and Markstein's correction of a reciprocal rounds it to nearest
but where the significand of the root is all ones, where it stays one unit below."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOW, HIGH = 2.0 ** -99, 2.0 ** 99  # the iteration's range


def _inputs(kind):
    rng = np.random.default_rng(5)
    if kind == "random":  # every exponent, random significands
        e = rng.integers(-1022, 1024, size=1 << 20)
        return np.ldexp(rng.uniform(1.0, 2.0, size=e.size), e)
    if kind == "pivots":  # 1 and below, as pivots of correlation matrices are
        return np.concatenate([10.0 ** -rng.uniform(0.0, 18.0, size=1 << 20), rng.uniform(size=1 << 20)])
    if kind == "ties":  # next to powers of two: roots and reciprocals closest to the middle of two numbers
        k = np.arange(1 << 14, dtype=np.int64)
        u = np.ldexp(1.0, np.arange(-6, 7)).view(np.int64)[:, None]
        return np.concatenate([u + k, u - k], axis=1).view(np.float64).ravel()
    k = np.arange(1 << 12, dtype=np.int64)
    t = np.array([LOW, HIGH, 1e-30, 1e30, 2.0 ** -1022]).view(np.int64)[:, None]
    special = np.array([0.0, 5e-324, 1e-310, np.finfo(float).max, np.inf])
    return np.concatenate([np.concatenate([t + k, t - k], axis=1).view(np.float64).ravel(), special])


@pytest.mark.parametrize("kind", ["random", "pivots", "ties", "thresholds"])
def test_equal_to_cuda(gpu_lib, kind):
    import libkriging_gb300 as lk
    x = np.ascontiguousarray(_inputs(kind))
    x = x[x >= 0.0]
    out = np.empty((4, x.size))
    dp = ctypes.POINTER(ctypes.c_double)
    assert lk.load().lkg_pivot_roots_check(x.size, x.ctypes.data_as(dp), out.ctypes.data_as(dp)) == 0
    root, rroot, root_c, rroot_c = out
    assert np.array_equal(root, root_c) and np.array_equal(root, np.sqrt(x))
    ones = (root.view(np.int64) & ((1 << 52) - 1)) == (1 << 52) - 1
    assert np.array_equal(rroot[~ones], rroot_c[~ones])
    off = rroot_c[ones].view(np.int64) - rroot[ones].view(np.int64)
    assert np.all((off == 0) | (off == 1))
