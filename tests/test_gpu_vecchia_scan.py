"""predictVecchia's FP32 neighbour scan and the local factorisation against the oracle: offsets that leave FP32
few digits, ties, the smallest and largest m, and blocks that the FP32 certificate cannot clear."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _model(lk, n, d, kernel, theta, shift=0.0, scale=1.0, seed=0, dup=0):
    rng = np.random.default_rng(seed)
    U = rng.uniform(size=(n, d))
    if dup:
        U[:, 0] = np.round(U[:, 0] * dup) / dup  # many equal distances
    X = shift + scale * U
    y = np.sin(2 * np.pi * U).sum(axis=1) + 0.1 * rng.standard_normal(n)
    th = np.full(d, theta * scale)
    k = lk.Kriging(kernel)
    k.fit(y, X, "constant", False, "none", "LL", {"theta": th.reshape(1, -1)})
    return k, X, y, th, shift + scale * rng.uniform(size=(70, d))


SHAPES = [(1, 2, 1), (40, 1, 32), (257, 2, 1), (300, 3, 31), (515, 5, 32), (400, 8, 17)]
SCALES = [(0.0, 1.0, 0), (1e5, 1.0, 0), (-3e7, 1e-2, 0), (0.0, 1e25, 0), (0.0, 1.0, 4)]


# (ties in d = 1 would be coincident points and a singular R)
@pytest.mark.parametrize("n,d,m,shift,scale,dup", [a + b for a in SHAPES for b in SCALES if not (a[1] == 1 and b[2])])
def test_predict_vecchia_vs_oracle(gpu_lib, n, d, m, shift, scale, dup):
    k, X, y, th, Xn = _model(gpu_lib, n, d, "matern3_2", 0.2, shift, scale, n + m, dup)
    mean, sd = k.predictVecchia(Xn, True, min(m, n))
    F = np.ones((n, 1))
    mo, so = O.predict_vecchia("matern3_2", X, y, F, k.beta(), th, k.sigma2(), Xn, np.ones((70, 1)), min(m, n))
    # equal sets give the repository's bounds; a shift of s leaves |x| / |dx| more rounding in every distance
    loss = 1.0 + abs(shift) / scale * 1e-2
    assert rel_err(mean, mo) < 1e-10 * loss and rel_err(sd, so) < 1e-8 * loss


@pytest.mark.parametrize("kernel,theta", [("exp", 0.05), ("exp", 5.0), ("gauss", 0.08), ("matern5_2", 0.5), ("matern3_2", 3.0)])
def test_vll_over_conditionings(gpu_lib, kernel, theta):
    """From blocks near the identity to blocks that the certificate leaves to the estimate."""
    rng = np.random.default_rng(4)
    X = rng.uniform(size=(350, 2))
    y = np.sin(2 * np.pi * X).sum(axis=1) + 0.1 * rng.standard_normal(350)
    k = gpu_lib.Kriging(kernel)
    k.set_vecchia_exact_commit(False)
    k.fit(y, X, "constant", False, "BFGS", "LLVecchia(32)", {"theta": np.full((1, 2), theta)})
    order, nbr = k.vecchia_sets()
    th = np.full(2, theta)
    v, g = k.logLikelihoodVecchiaFun(th, True)
    vo, go, _, _ = O.vecchia_ll(kernel, X, y, np.ones((350, 1)), th, order, nbr)
    # conditional variances down to 1 - r'a ~ 1 / cond(RN) carry cond eps
    RN = O.build_R(kernel, X[nbr[-1]], th)
    tol = max(1e-10, 64 * np.finfo(float).eps * np.linalg.cond(RN))
    assert rel_err(v, vo) < tol and rel_err(g, go) < 100 * tol
