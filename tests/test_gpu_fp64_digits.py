"""The FP64 path where its products run as digit products (n >= 192): panel, block and tile edges against the oracle."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _model(lk, n, d, kernel, nugget, seed, precision=0):
    rng = np.random.default_rng(seed)
    X = rng.uniform(size=(n, d))
    y = np.sin(2 * np.pi * X).sum(axis=1) + 0.1 * rng.standard_normal(n)
    th = rng.uniform(1.0, 2.0, size=d) * n ** (-1.0 / d)
    P = {"theta": th.reshape(1, -1)}
    if nugget:
        P.update(sigma2=1.0, nugget=1e-6)
    k = lk.Kriging(kernel, "nugget") if nugget else lk.Kriging(kernel)
    k.set_precision(precision)
    k.fit(y, X, "constant", False, "none", "LL", P)
    return k, X, y, th


@pytest.mark.parametrize("n", [191, 192, 193, 255, 256, 257, 319, 384, 513, 577, 1025])
@pytest.mark.parametrize("nugget", [False, True])
def test_loglik_at_block_edges(gpu_lib, n, nugget):
    k, X, y, th = _model(gpu_lib, n, 4, "matern5_2", nugget, n)
    g = np.append(th, 1.0 / (1.0 + 1e-6)) if nugget else th
    ll, grad, _ = k.logLikelihoodFun(g, True)
    assert k.last_slices() == 0
    ora = O.OracleKriging(y, X, "matern5_2", noise_model="nugget" if nugget else "none")
    ll_o, g_o = ora.log_likelihood(g)
    assert rel_err(ll, ll_o) < 1e-10 and rel_err(grad, g_o) < 1e-7


@pytest.mark.parametrize("n", [200, 300, 513])
def test_batched_bits_equal_single(gpu_lib, n):
    k, X, y, th = _model(gpu_lib, n, 3, "gauss", True, n)
    T = np.hstack([np.outer([0.7, 0.9, 1.0, 1.1, 1.2], th), np.full((5, 1), 0.999)])
    ll, grad = k.logLikelihoodFunBatch(T, True)
    for b in range(5):
        l1, g1, _ = k.logLikelihoodFun(T[b], True)
        assert l1 == ll[b] and np.array_equal(g1, grad[b])


@pytest.mark.parametrize("n", [193, 320, 520])
def test_loo_at_block_edges(gpu_lib, n):
    k, X, y, th = _model(gpu_lib, n, 3, "matern3_2", False, n)
    v, g = k.leaveOneOutFun(th, True)
    v_o, g_o = O.OracleKriging(y, X, "matern3_2").leave_one_out(th)[:2]
    assert rel_err(v, v_o) < 1e-9 and rel_err(g, g_o) < 1e-8


@pytest.mark.parametrize("n", [192, 300, 513])
@pytest.mark.parametrize("q", [16, 17, 32, 33, 129])
def test_predict_at_tile_edges(gpu_lib, n, q):
    k, X, y, th = _model(gpu_lib, n, 3, "matern5_2", False, n + q)
    Xn = np.random.default_rng(q).uniform(size=(q, 3))
    mean, sd, _, dm, ds = k.predict(Xn, True, False, True)
    ora = O.OracleKriging(y, X, "matern5_2")
    m = O.populate_model("matern5_2", ora.X, ora.y, ora.F, th, 1.0, None, False)
    mo, so, dmo, dso = ora.predict(Xn, th, m.betahat, m.SSEstar / n, return_deriv=True)
    assert rel_err(mean, mo) < 1e-9 and rel_err(sd, so) < 1e-7
    assert rel_err(dm, dmo) < 1e-9 and rel_err(ds, dso) < 1e-7


def test_long_products_in_chunks(gpu_lib):
    """64 matrices of 1100 rows: W^T W runs in chunks of 512 rows, the single matrix in one; the same bits."""
    k, X, y, th = _model(gpu_lib, 1100, 4, "matern5_2", True, 5)
    T = np.hstack([np.outer(np.linspace(0.8, 1.2, 64), th), np.full((64, 1), 0.999)])
    ll, grad = k.logLikelihoodFunBatch(T, True)
    for b in (0, 63):
        k1, _, _, _ = _model(gpu_lib, 1100, 4, "matern5_2", True, 5)
        l1, g1, _ = k1.logLikelihoodFun(T[b], True)
        assert l1 == ll[b] and np.array_equal(g1, grad[b])


@pytest.mark.parametrize("n", [200, 400])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_designs_are_refused(gpu_lib, n, bad):
    rng = np.random.default_rng(n)
    X, y = rng.uniform(size=(n, 3)), rng.standard_normal(n)
    X[5, 1] = bad
    k = gpu_lib.Kriging("matern5_2")
    with pytest.raises(gpu_lib.LibKrigingError):
        k.fit(y, X, "constant", False, "none", "LL", {"theta": np.full((1, 3), 0.3)})
