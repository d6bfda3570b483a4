"""Batches of many small matrices: digit scratch is shared by groups of entries, so a batch needs little more than its
matrices, and an entry's bits do not depend on the batch it is in."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(lk, n, d, nugget=False):
    rng = np.random.default_rng(n)
    X = rng.uniform(size=(n, d))
    k = lk.Kriging("matern5_2")
    k.fit(np.sin(4 * X).sum(axis=1) + 0.1 * rng.normal(size=n), X, optim="none", parameters={"theta": [[0.3] * d]})
    return k


@pytest.mark.parametrize("n,k", [(200, 1100), (193, 600), (520, 300)])
def test_groups_give_the_same_bits(gpu_lib, n, k):
    """More entries than one group of the panels (512 at n = 200) and of the long products (256) hold."""
    import libkriging_gb300 as lk
    th = np.random.default_rng(k).uniform(0.1, 0.5, size=(k, 2))
    ll, g = _model(lk, n, 2).logLikelihoodFunBatch(th, True)
    few = [0, 1, k // 2, k - 1]
    ll_f, g_f = _model(lk, n, 2).logLikelihoodFunBatch(th[few], True)
    assert np.array_equal(ll[few], ll_f) and np.array_equal(g[few], g_f)


def test_a_batch_fits_beside_its_matrices(gpu_lib):
    """1500 matrices of 200 rows take 1.7 GB with their inverses; 2.6 GB are enough for the evaluation."""
    import gc

    import torch

    import libkriging_gb300 as lk
    k, n = 1500, 200
    th = np.random.default_rng(1).uniform(0.1, 0.5, size=(k, 2))
    m = _model(lk, n, 2)
    few = [0, 700, k - 1]
    want = _model(lk, n, 2).logLikelihoodFunBatch(th[few], True)
    gc.collect()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - int(2.6e9), dtype=torch.uint8, device="cuda")
    try:
        ll, g = m.logLikelihoodFunBatch(th, True)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert np.array_equal(ll[few], want[0]) and np.array_equal(g[few], want[1])
