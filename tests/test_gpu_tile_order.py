"""Updates in tile order whose warps reach from one cluster to the next (their
points are walked one by one) against the oracle: two and more clusters far
apart with one outer dimension, sizes that are no multiples of 32, a few lone
points between them.

Counts and flags are exact by construction; a position is x + A / N with every
term below eps in magnitude and formed in FP32 with relative errors of a few
ulp, so 1e-5 absolute is far above the rounding at coordinates up to 1.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(n, d, clusters, spread, lone):
    rng = np.random.default_rng(n + d)
    c = np.linspace(0.06, 0.94, clusters)[rng.integers(0, clusters, n), None]
    X = c + spread * rng.standard_normal((n, d))
    X[:lone] = rng.random((lone, d))
    return np.clip(X, 0.0, 1.0).astype(np.float32)


@pytest.mark.parametrize("n,d,eps,clusters,spread,lone", [
    (16_389, 2, 0.009, 2, 0.02, 0),
    (16_389, 2, 0.009, 40, 0.002, 5),
    (17_001, 2, 0.004, 300, 0.001, 40),
    (16_401, 3, 0.006, 7, 0.01, 11),
    (16_401, 3, 0.0007, 500, 0.002, 300),
    (16_385, 4, 0.02, 60, 0.004, 3),
])
def test_step_matches_oracle(oracle, n, d, eps, clusters, spread, lone):
    from eggsync import egg_step

    X = points(n, d, clusters, spread, lone)
    xn, cnt, flags = egg_step(X, eps)
    oxn, ocnt, oflag = oracle.step(X, eps)
    assert np.array_equal(cnt, ocnt)
    assert flags[0] == oflag
    assert float(np.abs(xn - oxn).max()) <= 1e-5
