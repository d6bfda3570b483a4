"""The maxmin order in rounds of many steps against the one-step definition: ties, coincident points, sizes around the
candidate limit and launch boundaries."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _points(kind, n, d, rng):
    if kind == "uniform":
        return rng.uniform(size=(n, d))
    if kind == "lattice":  # distances tie by the thousand
        side = int(np.ceil(n ** (1.0 / d)))
        g = np.stack(np.meshgrid(*[np.arange(float(side))] * d), -1).reshape(-1, d)
        return g[rng.permutation(len(g))[:n]]
    if kind == "coincident":
        return np.round(rng.uniform(size=(n, d)) * 12) / 12
    if kind == "clusters":  # scales from 1 to 1e-12: FP32 differences say nothing about the innermost
        return np.concatenate([rng.normal(size=(n - 3 * (n // 4), d))] +
                              [0.3 + rng.normal(size=(n // 4, d)) * 10.0 ** -(4 * k) for k in (1, 2, 3)])
    return 1e8 + rng.uniform(size=(n, d)) * np.where(np.arange(d) == 0, 1.0, 1e-3)  # offset, one long axis


@pytest.mark.parametrize("kind", ["uniform", "lattice", "coincident", "clusters", "offset"])
@pytest.mark.parametrize("n,d", [(1, 1), (33, 1), (65, 2), (1025, 2), (2500, 3), (1500, 8)])
def test_order_equals_the_definition(gpu_lib, kind, n, d):
    import libkriging_gb300 as lk
    X = _points(kind, n, d, np.random.default_rng(n + d))
    order, nbr = lk.vecchia_sets(X, 5)
    order_o, nbr_o = O.vecchia_sets(X, 5)
    assert np.array_equal(order, order_o) and np.array_equal(nbr, nbr_o)


def test_launch_boundary(gpu_lib):
    """A second launch continues where the first one's last round was cut off; coincident points cross it too."""
    import libkriging_gb300 as lk
    rng = np.random.default_rng(8)
    X = np.concatenate([rng.uniform(size=(65000, 2)), np.repeat(rng.uniform(size=(50, 2)), 40, axis=0)])
    order, _ = lk.vecchia_sets(X, 1)
    assert np.array_equal(np.sort(order), np.arange(len(X)))
    # the 1950 repeated points come last, by ascending index, after every distinct one
    tail = order[-1950:]
    assert np.all(np.diff(tail) > 0) and tail.min() >= 65000
    # running distances of the order are non-increasing: checked on the last positions before the tail
    Z = X[order]
    r = [((Z[:t] - Z[t]) ** 2).sum(1).min() for t in range(65030, 65051)]
    assert np.all(np.diff(r) <= 0)
