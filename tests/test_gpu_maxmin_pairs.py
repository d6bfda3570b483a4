"""Maxmin rounds resolved from pairwise conflicts: every template of the dimension, boxes at and beyond the range of FP32
squares, and spacings where many candidates come down without leaving the round."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("scale", [1.0, 1e25, 1e-25, 1e15])
def test_dimensions_and_scales(gpu_lib, d, scale):
    import libkriging_gb300 as lk
    X = scale * np.random.default_rng(d).uniform(size=(1100, d))
    assert all(np.array_equal(a, b) for a, b in zip(lk.vecchia_sets(X, 4), O.vecchia_sets(X, 4)))


@pytest.mark.parametrize("amp", [0.0, 1e-9, 1e-4, 0.03, 0.1])
def test_jittered_lattice(gpu_lib, amp):
    """Distances within a few percent of one another: candidates come down to keys that still reach the threshold."""
    import libkriging_gb300 as lk
    rng = np.random.default_rng(3)
    g = np.stack(np.meshgrid(*[np.arange(15.0)] * 3), -1).reshape(-1, 3)[:2049]
    X = rng.permutation(g) + amp * rng.uniform(size=(2049, 3))
    assert all(np.array_equal(a, b) for a, b in zip(lk.vecchia_sets(X, 3), O.vecchia_sets(X, 3)))
