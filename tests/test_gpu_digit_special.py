"""Special values and every digit count of the digit-product kernel."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _product(lk, A, B, S):
    """A B^T with S digits on both tile widths (bit-identical by construction)."""
    lib = lk.load()
    (M, K), N = A.shape, B.shape[0]
    A, B = np.asfortranarray(A), np.asfortranarray(B)
    dp, ip = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)
    old, out = lib.lkg_get_digit_tile(), []
    try:
        for tn in (32, 64):
            assert lib.lkg_set_digit_tile(tn) == tn
            C, where = np.zeros((M, N), order="F"), np.zeros(8, dtype=np.int32)
            rc = lib.lkg_oz7_mode_check(0, M, N, K, A.ctypes.data_as(dp), B.ctypes.data_as(dp), S,
                                        C.ctypes.data_as(dp), where.ctypes.data_as(ip))
            assert rc == 0, (rc, where)
            out.append(C)
    finally:
        lib.lkg_set_digit_tile(old)
    assert np.array_equal(out[0], out[1], equal_nan=True)
    return out[0]


@pytest.mark.parametrize("S", [5, 6, 7, 8])
@pytest.mark.parametrize("shape", [(128, 32, 256), (130, 70, 64), (300, 129, 700)])
def test_infinities_and_nans_reach_their_rows_and_columns(gpu_lib, S, shape):
    """A row (column) with an infinity or NaN gives NaN in every product that reads it, and changes no other."""
    M, N, K = shape
    rng = np.random.default_rng(S)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((N, K))
    clean = _product(gpu_lib, A, B, S)
    # per term 2^-(7 S - 1) of either operand's truncation against the largest entries, plus the dropped digit pairs
    bound = K * 2.0 ** (4 - 7 * S) * np.abs(A).max() * np.abs(B).max() + 1e-15 * K * np.abs(A).max() * np.abs(B).max()
    assert np.abs(clean - A @ B.T).max() <= bound
    A[M - 1, K - 1], A[3, 0], B[N - 1, K // 2] = np.nan, np.inf, -np.inf
    got = _product(gpu_lib, A, B, S)
    bad = np.zeros((M, N), dtype=bool)
    bad[[3, M - 1], :] = True
    bad[:, N - 1] = True
    assert np.isnan(got[bad]).all()
    assert np.array_equal(got[~bad], clean[~bad])
