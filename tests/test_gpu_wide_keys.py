"""Updates of 4 < d <= 16 over the widths of a cell's key: 16 bits a dimension
up to d = 8, above that 8 or 16 bits on either side of 256 cells per dimension,
in single calls (against the oracle) and in batches that mix them (against
single calls: equal).

Counts and flags are exact by construction; a position is x + A / N with every
term below eps in magnitude and formed in FP32 with relative errors of a few
ulp, so 1e-5 absolute is far above the rounding at coordinates up to 1.
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(seed, n, d):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0.2, 0.8, (6, d))
    X = c[rng.integers(0, 6, n)] + 0.01 * rng.standard_normal((n, d))
    X[: n // 5] = rng.random((n // 5, d))
    X[n // 2: n // 2 + n // 8] = X[: n // 8]
    return np.clip(X, 0.0, 1.0).astype(np.float32)


def width(d, eps):
    side = np.float32(np.sqrt((float(np.float32(eps)) / 2) ** 2 / d))
    return int(np.float32(1.0) / side)


@pytest.mark.parametrize("n,d,eps,w", [
    (3_001, 5, 0.01, 447),
    (3_001, 6, 0.019, 257),
    (3_001, 7, 0.02, 264),
    (3_001, 8, 0.004, 1_414),
    (2_001, 9, 0.0233, 257),
    (2_001, 9, 0.0235, 255),
    (2_001, 14, 0.029, 258),
    (2_001, 16, 0.0311, 257),
    (2_001, 16, 0.0313, 255),
    (2_001, 16, 0.006, 1_333),
])
def test_step_matches_oracle(oracle, n, d, eps, w):
    from eggsync import egg_step

    assert width(d, eps) == w
    X = points(n + d, n, d)
    xn, cnt, flags = egg_step(X, eps)
    oxn, ocnt, oflag = oracle.step(X, eps)
    assert np.array_equal(cnt, ocnt)
    assert flags[0] == oflag
    assert float(np.abs(xn - oxn).max()) <= 1e-5


@pytest.mark.parametrize("spec", [
    [(3_000, 5, 0.01), (3_000, 5, 0.0244), (70, 5, 0.08)],
    [(2_000, 16, 0.02), (2_500, 16, 0.15), (33, 16, 0.0312)],
    [(2_000, 12, 0.02), (2_500, 12, 0.1), (1_000, 24, 0.3), (900, 7, 0.02)],
])
def test_mixed_batch_equals_single_runs(spec):
    from eggsync import egg_sync, egg_sync_batch

    inst = [(points(k, n, d), eps) for k, (n, d, eps) in enumerate(spec)]
    out, _ = egg_sync_batch(inst)
    for (X, eps), (labels, info) in zip(inst, out):
        s_labels, s_info = egg_sync(X, eps)
        assert np.array_equal(labels, s_labels) and info["iterations"] == s_info["iterations"]


def test_batch_with_more_points_a_block():
    """606,208 points and more of one dimension: 32 a block in the batch, 16 in single calls."""
    from eggsync import egg_sync, egg_sync_batch

    inst = [(points(k, 325_001, 5), eps) for k, eps in enumerate((0.012, 0.03))]
    out, _ = egg_sync_batch(inst, max_iter=3, tune="off")
    for (X, eps), (labels, info) in zip(inst, out):
        s_labels, s_info = egg_sync(X, eps, max_iter=3)
        assert np.array_equal(labels, s_labels) and info["iterations"] == s_info["iterations"]


def test_one_narrow_eps_does_not_slow_its_batch():
    """An instance with more than 256 cells per dimension costs its batch what
    it costs by itself: it used to take every instance of its dimension to the
    kernel for any d (4.8 times slower)."""
    import torch
    from eggsync import egg_sync_batch

    X = torch.from_numpy(points(1, 20_000, 5)).cuda()

    def ms(eps):
        inst = [(X, e) for e in eps]
        out = [torch.empty(len(X), dtype=torch.int32, device="cuda") for _ in inst]
        egg_sync_batch(inst, max_iter=4, tune="off", labels_out=out)
        t = []
        for _ in range(5):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            egg_sync_batch(inst, max_iter=4, tune="off", labels_out=out)
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        return min(t)

    wide = [0.04, 0.05, 0.06, 0.07] * 4
    assert ms(wide + [0.012]) < 2 * ms(wide + [0.04])
