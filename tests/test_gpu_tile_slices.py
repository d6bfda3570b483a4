"""Covariances and gradient sums of matrices whose tiles are cut into slices (few tiles) and of those that are not."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["gauss", "exp", "matern5_2"])
@pytest.mark.parametrize("n,d", [(3, 2), (64, 5), (65, 3), (129, 9), (190, 20), (511, 4), (641, 4), (1020, 3)])
def test_loglik_around_the_slice_counts(gpu_lib, kernel, n, d):
    rng = np.random.default_rng(n)
    X = rng.uniform(size=(n, d))
    y = np.sin(2 * np.pi * X).sum(axis=1) + 0.1 * rng.standard_normal(n)
    th = rng.uniform(0.8, 1.4, size=d) * n ** (-1.0 / d)
    k = gpu_lib.Kriging(kernel)
    k.fit(y, X, "constant", False, "none", "LL", {"theta": th.reshape(1, -1)})
    ll, g, _ = k.logLikelihoodFun(th, True)
    ll_o, g_o = O.OracleKriging(y, X, kernel).log_likelihood(th)
    assert rel_err(ll, ll_o) < 1e-10 and rel_err(g, g_o) < 1e-7
    # and a batch gives the same bits
    llb, gb = k.logLikelihoodFunBatch(np.vstack([th, 1.1 * th, th]), True)
    assert llb[0] == ll and llb[2] == ll and np.array_equal(gb[0], g) and np.array_equal(gb[2], g)
    # covariances: rectangles of few and many tiles
    for q in (1, 70, 700):
        Z = rng.uniform(size=(q, d))
        C = k.covMat(X, Z)
        assert rel_err(C, k.sigma2() * O.cov_cross(kernel, X, Z, th)) < 1e-13
