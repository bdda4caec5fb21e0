"""d = 7 runs the generic kernels, which keep a point's sin and 1 - cos offsets
in arrays of their own: they must not share memory (the packed records of the
other d <= 8 leave those arrays empty)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_step_matches_oracle(oracle):
    from eggsync import egg_step

    rng = np.random.default_rng(7)
    c = rng.uniform(0.2, 0.8, (5, 7))
    X = np.clip(c[rng.integers(0, 5, 5000)] + 0.02 * rng.standard_normal((5000, 7)), 0, 1).astype(np.float32)
    xn, cnt, flags = egg_step(X, 0.05)
    oxn, ocnt, oflag = oracle.step(X, 0.05)
    assert np.array_equal(cnt, ocnt)
    assert flags[0] == oflag
    assert float(np.abs(xn - oxn).max()) <= 1e-5
