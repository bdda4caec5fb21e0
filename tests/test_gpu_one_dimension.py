"""One update of one-dimensional points against the oracle: cells of one to a
few groups of 32 points, of just under, exactly and over 32 groups (the groups
of a large cell are screened 32 at a time), points outside [0, 1] and repeated
points.

Counts and flags are exact by construction; a position is x + A / N with every
term below eps in magnitude and formed in FP32 with relative errors of a few
ulp, so 1e-5 absolute is far above the rounding at coordinates up to 1.2.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(n, lo=0.0, hi=1.0):
    rng = np.random.default_rng(n)
    X = rng.choice([0.31, 0.352, 0.7], n)[:, None] + 0.02 * rng.standard_normal((n, 1))
    X[: n // 8] = rng.uniform(lo, hi, (n // 8, 1))
    return np.clip(X, lo, hi).astype(np.float32)


def one_cell(m, n):
    """m points inside one cell of eps 0.1 (side 0.05), the others spread to its left and right."""
    rng = np.random.default_rng(m)
    X = rng.uniform(0.0, 1.0, (n, 1))
    X[:m] = rng.uniform(0.5001, 0.5499, (m, 1))
    return X.astype(np.float32)


@pytest.mark.parametrize("X,eps", [
    (points(33), 0.1),
    (points(2_001), 0.1),
    (points(20_003), 0.1),
    (points(20_003), 0.003),
    (points(30_000, -0.2, 1.2), 0.05),
    (one_cell(992, 3_000), 0.1),
    (one_cell(1_024, 3_000), 0.1),
    (one_cell(1_056, 3_000), 0.1),
    (one_cell(2_080, 2_200), 0.1),
    (points(40_000)[np.random.default_rng(1).integers(0, 300, 40_000)], 0.06),
])
def test_step_matches_oracle(oracle, X, eps):
    from eggsync import egg_step

    xn, cnt, flags = egg_step(X, eps)
    oxn, ocnt, oflag = oracle.step(X, eps)
    assert np.array_equal(cnt, ocnt)
    assert flags[0] == oflag
    lone = ocnt == 0  # beyond its clamped cell's box: 0 / 0 on both sides
    assert np.array_equal(np.isnan(xn[:, 0]), lone) and np.array_equal(np.isnan(oxn[:, 0]), lone)
    assert float(np.abs(xn - oxn)[~lone].max()) <= 1e-5


def test_batch_equals_single_runs():
    from eggsync import egg_sync, egg_sync_batch

    inst = [(points(n), eps) for n, eps in ((20_003, 0.1), (33, 0.05), (5_000, 0.004), (9_999, 0.02))]
    out, _ = egg_sync_batch(inst)
    for (X, eps), (labels, info) in zip(inst, out):
        s_labels, s_info = egg_sync(X, eps)
        assert np.array_equal(labels, s_labels) and info["iterations"] == s_info["iterations"]
