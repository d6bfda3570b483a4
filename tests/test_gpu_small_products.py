"""Products of few tiles (one entry per thread) against the oracle, and against the large tiles that a big batch takes: the
same bits."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65, 72, 127, 129, 150, 191])
def test_few_and_many_tiles(gpu_lib, n):
    rng = np.random.default_rng(n)
    X = rng.uniform(size=(n, 3))
    y = np.sin(2 * np.pi * X).sum(axis=1) + 0.1 * rng.standard_normal(n)
    th = np.array([0.3, 0.5, 0.4])
    k = gpu_lib.Kriging("matern5_2")
    k.fit(y, X, "linear", False, "none", "LL", {"theta": th.reshape(1, -1)})
    ll, g, _ = k.logLikelihoodFun(th, True)
    ora = O.OracleKriging(y, X, "matern5_2", "linear")
    ll_o, g_o = ora.log_likelihood(th)
    assert rel_err(ll, ll_o) < 1e-10 and rel_err(g, g_o) < 1e-7
    T = np.vstack([th] + [th * rng.uniform(0.7, 1.3, size=3) for _ in range(399)])  # 400 matrices: no product is small
    llb, gb = k.logLikelihoodFunBatch(T, True)
    assert llb[0] == ll and np.array_equal(gb[0], g)
    for q in (17, 1000):  # many right-hand sides
        Z = rng.uniform(size=(q, 3))
        m, s = k.predict(Z, True, False, False)[:2]
        m_o, s_o = ora.predict(Z, th, k.beta(), k.sigma2())[:2]
        assert rel_err(m, m_o) < 1e-9 and np.max(np.abs(s - s_o)) < 1e-7
