"""The maxmin order of boxes whose sides are small, where squares of FP32 quantities underflow: lattices whose points are
moved by 3e-6 to 3e-5 of the spacing, which is within the error of FP32 differences of such sides, against the one-step
definition."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [1.0, 1e-15, 2e-16, 1e-16, 5e-17, 2e-17, 5e-18, 1.5e-18, 5e-19])
@pytest.mark.parametrize("jitter", [3e-6, 1e-5, 3e-5])
def test_jittered_lattice(gpu_lib, side, jitter):
    import libkriging_gb300 as lk
    rng = np.random.default_rng(7)
    g = np.stack(np.meshgrid(np.arange(100.0), np.arange(100.0)), -1).reshape(-1, 2)
    X = side / 100 * rng.permutation(g + jitter * rng.uniform(size=g.shape))
    assert np.array_equal(lk.vecchia_sets(X, 1)[0], O.vecchia_sets(X, 1)[0])


@pytest.mark.parametrize("d", [3, 4, 6])
def test_dimensions(gpu_lib, d):
    import libkriging_gb300 as lk
    rng = np.random.default_rng(d)
    g = np.stack(np.meshgrid(*[np.arange({3: 14.0, 4: 7.0, 6: 4.0}[d])] * d), -1).reshape(-1, d)
    X = 2e-18 * rng.permutation(g + 1e-5 * rng.uniform(size=g.shape))
    assert np.array_equal(lk.vecchia_sets(X, 1)[0], O.vecchia_sets(X, 1)[0])
