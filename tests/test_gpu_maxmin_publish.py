"""Every step of a round is carried out, also the last ones before a launch or a round ends: short orders of many sizes,
each a permutation that equals the one-step definition where the oracle is quick."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3])
def test_no_step_is_lost_at_the_end(gpu_lib, d):
    import libkriging_gb300 as lk
    rng = np.random.default_rng(d)
    for n in rng.integers(2, 3000, size=120):
        X = rng.uniform(size=(int(n), d))
        order, _ = lk.vecchia_sets(X, 1)
        assert np.array_equal(np.sort(order), np.arange(n))
        if n <= 600:
            assert np.array_equal(order, O.vecchia_sets(X, 1)[0])
