"""A digit product whose wait expires is reported by the model that ran it, once, and by no other: its engines' status words
are set as the kernel sets them."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(lk, seed, n=300):
    rng = np.random.default_rng(seed)
    X = rng.uniform(size=(n, 2))
    k = lk.Kriging("matern5_2")
    k.fit(np.sin(5 * X).sum(axis=1) + 0.1 * rng.normal(size=n), X, optim="none", parameters={"theta": [[0.3, 0.3]]})
    return k


def _mark(lk, k):
    assert lk.load().lkg_kriging_mark_digits_expired(k._h) == 0


def test_only_the_failing_model_reports(gpu_lib, tmp_path):
    import libkriging_gb300 as lk
    a, b = _model(lk, 1), _model(lk, 2)
    th = np.array([0.25, 0.35])
    calls = [lambda k: k.logLikelihoodFun(th, return_grad=True), lambda k: k.logLikelihoodFun(th, return_grad=False),
             lambda k: k.leaveOneOutFun(th, return_grad=True), lambda k: k.save(str(tmp_path / "m.json"))]
    for call in calls:
        want = call(b)
        call(a)
        _mark(lk, a)
        again = call(b)
        with pytest.raises(Exception, match="timed out"):
            call(a)
        call(a)  # reported once
        if want is not None:
            assert all(np.array_equal(np.asarray(x), np.asarray(y)) for x, y in zip(want, again) if x is not None)
        a, b = _model(lk, 1), _model(lk, 2)


def test_models_in_threads(gpu_lib):
    import libkriging_gb300 as lk
    a, b = _model(lk, 1), _model(lk, 2)
    th = np.array([0.25, 0.35])
    a.logLikelihoodFun(th, return_grad=True)
    want = b.logLikelihoodFun(th, return_grad=True)

    def failing():
        n = 0
        for _ in range(30):
            _mark(lk, a)
            try:
                a.logLikelihoodFun(th, return_grad=True)
            except Exception as e:
                n += "timed out" in str(e)
        return n

    def healthy():
        return [b.logLikelihoodFun(th, return_grad=True) for _ in range(60)]

    with ThreadPoolExecutor(2) as ex:
        f, h = ex.submit(failing), ex.submit(healthy)
        assert f.result() == 30
        assert all(ll == want[0] and np.array_equal(g, want[1]) for ll, g, *_ in h.result())
