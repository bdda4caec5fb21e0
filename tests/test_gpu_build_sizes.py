"""The grid build against the oracle where it changes path: one block, a cluster
of 8 and of 16 blocks, the per-pass launches beyond; keys of one to several
words, more than 256 cells per dimension, no outer dimension.  Integers: equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [
    (1, 3, 0.1), (2, 2, 0.05), (33, 4, 0.05), (1_024, 3, 0.05), (1_025, 3, 0.05), (1_025, 1, 0.0004),
    (5_000, 2, 0.004), (5_000, 9, 0.1), (16_384, 3, 0.03), (16_385, 5, 0.05), (20_000, 16, 0.15), (3_000, 33, 0.4),
    (131_072, 3, 0.02), (131_073, 3, 0.02), (131_073, 2, 0.003),
]


def points(n, d):
    rng = np.random.default_rng(n + d)
    c = rng.uniform(0.2, 0.8, (7, d))
    X = np.clip(c[rng.integers(0, 7, n)] + 0.05 * rng.standard_normal((n, d)), 0, 1).astype(np.float32)
    X[n // 2:] = X[: n - n // 2]  # equal keys: the order is by index
    return X


@pytest.mark.parametrize("n,d,eps", SIZES)
def test_grid_matches_oracle(oracle, n, d, eps):
    from eggsync import egg_grid

    X = points(n, d)
    order, cell_of, start = egg_grid(X, eps)
    o_order, o_cell_of, o_start = oracle.grid(X, eps)
    assert np.array_equal(order, o_order)
    assert np.array_equal(start, o_start)
    assert np.array_equal(cell_of, o_cell_of[o_order])


@pytest.mark.parametrize("sizes", [SIZES[:4], SIZES[4:12], SIZES[:12] + SIZES[13:14]])
def test_batch_equals_single_runs(sizes):
    from eggsync import egg_sync, egg_sync_batch

    out, _ = egg_sync_batch([(points(n, d), eps) for n, d, eps in sizes], max_iter=6)
    for (n, d, eps), (labels, info) in zip(sizes, out):
        s_labels, s_info = egg_sync(points(n, d), eps, max_iter=6)
        assert np.array_equal(labels, s_labels) and info["iterations"] == s_info["iterations"]
