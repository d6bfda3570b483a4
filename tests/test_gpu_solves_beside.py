"""Evaluations with gradient run their solves beside the inverse: the same bits as stage by stage, also when the first
factorisation fails and is redone with the numerical nugget, and in batches whose entries fail one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trend", ["none", "linear"])
@pytest.mark.parametrize("n", [7, 63, 64, 65, 191, 257, 700])
def test_same_bits_as_stage_by_stage(gpu_lib, n, trend):
    rng = np.random.default_rng(n)
    X = rng.uniform(size=(n, 3))
    if n > 63:
        X[n // 2] = X[3]  # a coincident pair: the first factorisation fails or is rejected by its rcond
    y = np.sin(4 * X).sum(axis=1)
    k = gpu_lib.Kriging("matern5_2")
    th = np.full(X.shape[1], 0.4)
    k.fit(y, X, trend, False, "none", "LL", {"theta": th.reshape(1, -1)})
    staged = k.logLikelihoodFun(th, True, bench=True)
    for _ in range(3):  # direct, captured, replayed
        ll, g, _ = k.logLikelihoodFun(th, True)
        assert ll == staged[0] and np.array_equal(g, staged[1])
    T = np.vstack([th, 0.3 * th, 1.2 * th])
    llb, gb = k.logLikelihoodFunBatch(T, True)
    for i, t in enumerate(T):
        ll, g, _ = k.logLikelihoodFun(t, True, bench=True)
        assert llb[i] == ll and np.array_equal(gb[i], g)
