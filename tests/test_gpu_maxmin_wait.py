"""The waits inside the maxmin kernel end: with no patience the call reports it, and the next call is sound."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out_is_an_error(gpu_lib):
    import libkriging_gb300 as lk
    lib = lk.load()
    X = np.asfortranarray(np.random.default_rng(1).uniform(size=(3000, 2)))
    order = np.empty(len(X), dtype=np.int32)

    def call(ns):
        return lib.lkg_vecchia_sets_wait_check(len(X), 2, X.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), ns,
                                               order.ctypes.data_as(ctypes.POINTER(ctypes.c_int)))

    assert call(0) == -1  # gives up at the first step that is not there yet
    assert b"timed out" in lib.lkg_get_last_error()
    assert call(1_000_000_000) == 0
    assert np.array_equal(order, O.vecchia_sets(X, 1)[0])
