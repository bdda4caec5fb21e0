"""One update against the oracle where its walks change path: around the size
from which the points are put in tile order, one to four outer dimensions,
more than 256 cells per dimension, points outside [0, 1] (clamped into the
grid's edge cells), collapsed points, and d above 4 with one byte per cell
coordinate (width <= 256) and without.

Counts and flags are exact by construction; a position is x + A / N with every
term below eps in magnitude and formed in FP32 with relative errors of a few
ulp, so 1e-5 absolute is far above the rounding at coordinates up to 1.2.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(seed, n, d, lo=0.0, hi=1.0, dup=False):
    rng = np.random.default_rng(seed)
    k = 6
    c = rng.uniform(0.2, 0.8, (k, d))
    X = c[rng.integers(0, k, n)] + 0.03 * rng.standard_normal((n, d))
    noise = rng.random(n) < 0.2
    X[noise] = rng.uniform(lo, hi, (int(noise.sum()), d))
    if dup:
        X = X[rng.integers(0, n // 8, n)]
    return np.clip(X, lo, hi).astype(np.float32)


@pytest.mark.parametrize("n,d,eps,lo,hi,dup", [
    (16_383, 3, 0.05, 0.0, 1.0, False),
    (16_384, 3, 0.05, 0.0, 1.0, False),
    (16_385, 3, 0.05, -0.2, 1.2, False),
    (16_400, 2, 0.05, -0.2, 1.2, False),
    (16_400, 2, 0.009, 0.0, 1.0, False),   # one outer dimension, width 314
    (16_400, 3, 0.15, 0.0, 1.0, False),    # three outer dimensions
    (16_400, 4, 0.35, 0.0, 1.0, False),    # four outer dimensions
    (16_400, 4, 0.08, -0.1, 1.1, False),
    (20_011, 3, 0.03, 0.0, 1.0, True),
    (16_400, 3, 0.006, 0.0, 1.0, False),   # width 577
    (3_001, 5, 0.1, -0.1, 1.1, False),
    (3_001, 5, 0.016, 0.0, 1.0, False),    # width 279: no byte keys
    (3_001, 8, 0.2, 0.0, 1.0, False),
    (2_001, 14, 0.2, 0.0, 1.0, False),
    (2_001, 16, 0.2, -0.1, 1.1, False),
    (2_001, 17, 0.2, 0.0, 1.0, False),
])
def test_step_matches_oracle(oracle, n, d, eps, lo, hi, dup):
    from eggsync import egg_step

    X = points(n + d, n, d, lo, hi, dup)
    xn, cnt, flags = egg_step(X, eps)
    oxn, ocnt, oflag = oracle.step(X, eps)
    assert np.array_equal(cnt, ocnt)
    assert flags[0] == oflag
    # a point beyond its clamped cell's box has no neighbour at all: 0 / 0 on both sides
    lone = ocnt == 0
    assert np.array_equal(np.isnan(xn), np.repeat(lone[:, None], d, 1))
    assert np.array_equal(np.isnan(oxn), np.isnan(xn))
    assert float(np.abs(xn - oxn)[~lone].max()) <= 1e-5
