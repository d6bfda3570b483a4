"""The digit solves of a prediction take a bounded number of points at a time: scratch stays small beside the chunk's
covariances, and the points' results do not depend on the split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(lk, n=200, d=2):
    rng = np.random.default_rng(4)
    X = rng.uniform(size=(n, d))
    k = lk.Kriging("matern5_2")
    k.fit(np.sin(5 * X).sum(axis=1) + 0.1 * rng.normal(size=n), X, optim="none", parameters={"theta": [[0.3] * d]})
    return k


def test_points_across_the_split(gpu_lib):
    import libkriging_gb300 as lk
    k = _model(lk)
    X = np.random.default_rng(5).uniform(size=(16384 * 2 + 33, 2))
    mean, sd = k.predict(X, True, False, False)[:2]
    for lo, hi in ((0, 50), (16350, 16420), (32760, len(X))):
        m, s = k.predict(X[lo:hi], True, False, False)[:2]
        assert np.array_equal(mean[lo:hi], m) and np.array_equal(sd[lo:hi], s)


def test_scratch_beside_the_covariances(gpu_lib):
    """150000 points on 200: 240 MB of covariances and some 20 MB for the points; 0.5 GB must do."""
    import gc

    import torch

    import libkriging_gb300 as lk
    k = _model(lk)
    X = np.random.default_rng(6).uniform(size=(150000, 2))
    want = k.predict(X[:100], True, False, False)[:2]
    gc.collect()
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - int(0.5e9), dtype=torch.uint8, device="cuda")
    try:
        mean, sd = k.predict(X, True, False, False)[:2]
    finally:
        del hold
        torch.cuda.empty_cache()
    assert np.array_equal(mean[:100], want[0]) and np.array_equal(sd[:100], want[1])
