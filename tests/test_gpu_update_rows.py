"""Gathered points: rows of columns, joint walks across columns, several rows of
points per warp.  Results must equal the full recomputation bit for bit, and
one update's counts the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def gathered(n, d, spots, seed):
    rng = np.random.default_rng(seed)
    c = rng.random((spots, d)).astype(np.float32)
    X = c[rng.integers(0, spots, n)]
    k = n // 50  # some that still move, some alone
    X[:k] = np.clip(X[:k] + 0.02 * rng.standard_normal((k, d)), 0, 1)
    X[k: k + k // 4] = rng.random((k // 4, d))
    return X[rng.permutation(n)].astype(np.float32)


# one row per warp (up to 94,720 points), two, three, the most (8 from 663,041 points on)
@pytest.mark.parametrize("n,d,eps,spots", [
    (20_000, 1, 0.002, 40), (20_000, 2, 0.05, 40), (94_720, 2, 0.03, 300), (94_721, 3, 0.05, 300),
    (200_001, 4, 0.06, 500), (300_033, 3, 0.02, 5_000), (800_007, 3, 0.015, 20_000),
])
def test_incremental_equals_full(n, d, eps, spots):
    from eggsync import egg_sync

    X = gathered(n, d, spots, n)
    out = []
    for full in (False, True):
        pos = np.empty_like(X)
        labels, info = egg_sync(X, eps, max_iter=25, full_update=full, positions_out=pos)
        out.append((labels, pos, info["iterations"]))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][2] == out[1][2]
    assert np.array_equal(out[0][1].view(np.int32), out[1][1].view(np.int32))


@pytest.mark.parametrize("n,d,eps,spots", [(20_000, 2, 0.05, 40), (30_000, 3, 0.04, 200), (20_000, 4, 0.1, 3_000)])
def test_step_counts_match_oracle(oracle, n, d, eps, spots):
    from eggsync import egg_step

    X = gathered(n, d, spots, d)
    xn, cnt, flags = egg_step(X, eps)
    oxn, ocnt, oflag = oracle.step(X, eps)
    assert np.array_equal(cnt, ocnt)
    assert flags[0] == oflag
    assert np.abs(xn - oxn).max() <= 1e-5
