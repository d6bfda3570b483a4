"""Rounding of the covariance values from five dimensions on, where the plain product form loses digits: root mean square of
the relative errors against extended precision, beside what the log1p form has in FP64 arithmetic on the same pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forms(kernel, B, theta):
    """(extended precision, log1p form in FP64) of the points B against the origin."""
    out = []
    for T in (np.longdouble, np.float64):
        t = np.abs(B.astype(T)) / T(theta)
        if kernel == "gauss":
            out.append(np.exp(-(t * t).sum(1) / 2))
        elif kernel == "exp":
            out.append(np.exp(-t.sum(1)))
        else:
            t = np.sqrt(T(3 if kernel == "matern3_2" else 5)) * t
            s = T(0) * t[:, 0]
            for k in range(t.shape[1]):  # as it is summed on the device
                s = s + (t[:, k] - np.log1p(t[:, k] if kernel == "matern3_2" else t[:, k] + t[:, k] * t[:, k] / T(3)))
            out.append(np.exp(-s))
    return out


@pytest.mark.parametrize("kernel", ["gauss", "exp", "matern3_2", "matern5_2"])
@pytest.mark.parametrize("d", [5, 8, 9, 16])
@pytest.mark.parametrize("theta", [0.05, 0.3, 1.0, 3.0, 10.0])
def test_no_larger_than_the_log1p_forms(gpu_lib, kernel, d, theta):
    import libkriging_gb300 as lk
    rng = np.random.default_rng(d)
    X, y = rng.uniform(size=(40, d)), rng.standard_normal(40)
    k = lk.Kriging(kernel)
    k.fit(y, X, "constant", False, "none", "LL",
          {"theta": np.full((1, d), theta), "sigma2": 1.0, "is_sigma2_estim": False})
    B = rng.uniform(size=(20000, d))
    got = k.covMat(np.zeros((1, d)), B)[0]
    want, ref = _forms(kernel, B, theta)
    near = want > 1e-290  # normal numbers
    rms = [np.sqrt(np.mean((((v.astype(np.longdouble) - want) / want)[near].astype(float) * 2.0 ** 53) ** 2))
           for v in (got, ref)]
    # beside the log1p form's: CUDA's exponential, good to one unit in the last place, and one more rounding, together below
    # one unit of 2^-53 (rms 0.6 each); a tenth for the scale sqrt(3) / theta or sqrt(5) / theta, rounded once for all pairs
    assert rms[0] <= np.hypot(1.1 * rms[1], 0.85), rms
