"""A part of the loop graph that cannot be captured (injected on the host, no
GPU fault): the call drives its loop from the host with the same results, the
stream is not left in capture, and the next call captures its graph again."""
import numpy as np
import pytest

from eggsync import _lib, egg_sync, egg_sync_batch

pytestmark = pytest.mark.gpu


def points(n, d, seed):
    rng = np.random.default_rng(seed)
    X = rng.uniform(0.2, 0.8, (5, d))[rng.integers(0, 5, n)] + 0.04 * rng.standard_normal((n, d))
    return np.clip(X, 0, 1).astype(np.float32)


@pytest.mark.parametrize("n", [3_000, 140_000])
def test_single_call(eggsync_lib, n):
    X = points(n, 3, n)
    ref, ri = egg_sync(X, 0.06)
    assert eggsync_lib.egg_release() == _lib.EGG_OK
    assert eggsync_lib.egg_inject_capture_failures(1) == _lib.EGG_OK
    for _ in range(2):
        lab, info = egg_sync(X, 0.06)
        assert np.array_equal(lab, ref) and info["iterations"] == ri["iterations"]
    assert eggsync_lib.egg_inject_capture_failures(0) == _lib.EGG_OK


def test_batch(eggsync_lib):
    inst = [(points(2_000, 2, 1), 0.05), (points(900, 5, 2), 0.1), (points(1_500, 2, 3), 0.03)]
    ref, _ = egg_sync_batch(inst, tune="off")
    assert eggsync_lib.egg_release() == _lib.EGG_OK
    assert eggsync_lib.egg_inject_capture_failures(1) == _lib.EGG_OK
    for _ in range(2):
        got, _ = egg_sync_batch(inst, tune="off")
        for (a, ia), (b, ib) in zip(got, ref):
            assert np.array_equal(a, b) and ia["iterations"] == ib["iterations"]
    assert eggsync_lib.egg_inject_capture_failures(0) == _lib.EGG_OK
