"""The covariance kernels over the exponential's whole range: product form against extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def exact(kernel, t):
    """C from the scaled distances t (rows: pairs), in extended precision through the logarithm."""
    t = np.abs(t).astype(np.longdouble)
    if kernel == "gauss":
        return np.exp(-(t * t).sum(1) / 2)
    if kernel == "exp":
        return np.exp(-t.sum(1))
    if kernel == "matern3_2":
        t = np.sqrt(np.longdouble(3)) * t
        return np.exp((np.log1p(t) - t).sum(1))
    t = np.sqrt(np.longdouble(5)) * t
    return np.exp((np.log1p(t + t * t / 3) - t).sum(1))


@pytest.mark.parametrize("kernel", ["gauss", "exp", "matern3_2", "matern5_2"])
@pytest.mark.parametrize("d", [1, 4, 7, 32])
def test_covariance_over_the_exponent_range(gpu_lib, kernel, d):
    import libkriging_gb300 as lk
    rng = np.random.default_rng(d)
    n = 70  # one full 64-wide tile and a ragged one
    X, y = rng.uniform(size=(n, d)), rng.standard_normal(n)
    k = lk.Kriging(kernel)
    k.fit(y, X, "constant", False, "none", "LL", {"theta": np.full((1, d), 0.3), "sigma2": 1.0, "is_sigma2_estim": False})
    # one point against points at growing distances: exponent sums 1e-3 .. 2500, across 700 and 1500
    sums = np.concatenate([np.geomspace(1e-3, 650, 40), np.linspace(690, 760, 30), np.linspace(1400, 2500, 30)])
    scale = {"gauss": 1.0, "exp": 1.0, "matern3_2": np.sqrt(3.0), "matern5_2": np.sqrt(5.0)}[kernel]
    w = rng.uniform(0.5, 1.0, size=(sums.size, d))
    t = w * (np.sqrt(2 * sums / (w * w).sum(1)) if kernel == "gauss" else sums / w.sum(1) / scale)[:, None]
    B = t * 0.3
    got = k.covMat(np.zeros((1, d)), B)[0]
    want = exact(kernel, B.astype(np.longdouble) / np.longdouble(0.3))
    # rounding of each scaled distance (3 eps) and of the d-term sum enters the exponent; the product adds 4 per factor
    tol = EPS * ((d + 3) * np.minimum(sums, 800) * 1.01 + 4 * d + 8)
    err = np.abs((got.astype(np.longdouble) - want)).astype(np.float64)
    assert np.all(err <= tol * want.astype(np.float64) + 2 * 4.95e-324 + 2.3e-308 * EPS * 64)
    assert np.all(got[sums > 1600] == want[sums > 1600].astype(np.float64))


@pytest.mark.parametrize("kernel", ["matern3_2", "matern5_2"])
def test_infinite_distances_are_not_zero_covariances(gpu_lib, kernel):
    import libkriging_gb300 as lk
    rng = np.random.default_rng(3)
    X, y = rng.uniform(size=(9, 2)), rng.standard_normal(9)
    k = lk.Kriging(kernel)
    k.fit(y, X, "constant", False, "none", "LL", {"theta": np.full((1, 2), 0.3)})
    assert np.isnan(k.covMat(np.zeros((1, 2)), np.array([[np.inf, 0.0], [np.nan, 0.1]]))).all()
