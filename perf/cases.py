"""What a user of eggsync has it do, as cases that can be timed one by one.

``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges,
``prepare(case, seed)`` the inputs a program holds before the call,
``run(state)`` one pass through the package's public entry points,
``work(case)`` the bytes and operations a pass cannot do without and
``exact(case, seed)`` its computed numbers in 64 bits, by plain torch.

Points are Gaussian blobs over uniform noise, min-max normalised: the shapes
of ``eggsync.data`` (10,000 x 2 up to 1,000,000 x 3, 20,000 x 16, the rows of
the reference's real data sets, the eps sweep over d = 2, 3 and 5).
"""
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

PKG = Path(__file__).resolve().parent.parent / "egg-sync_b200"
if str(PKG) not in sys.path:
    sys.path.insert(0, str(PKG))

import eggsync  # noqa: E402
from eggsync import data, warm  # noqa: E402

LAMBDA = data.LAMBDA
F32 = np.float32


def _cluster(name, n, d, eps, clusters, std_lo, std_hi, noise, io="device", stop="flag", **more):
    return dict(name=name, kind="cluster", n=n, d=d, eps=eps, clusters=clusters, std_lo=std_lo, std_hi=std_hi,
                noise=noise, io=io, stop=stop, **more)


def listed():
    return [
        # the smallest data set of the reference's experiments, through the
        # drop-in wrapper and host tensors: call latency and launches count
        _cluster("dropin_150x4", 150, 4, 0.05, 8, 0.02, 0.08, 0.05, io="dropin"),
        # the ordinary small run of the reference's synthetic experiments
        _cluster("cluster_10kx2", 10_000, 2, 0.05, 10, 0.02, 0.02, 0.05),
        # a middle-sized real data set (odd row count), host in, host out
        _cluster("dropin_45781x3", 45_781, 3, 0.05, 8, 0.02, 0.08, 0.05, io="dropin"),
        # high-dimensional rows (letter recognition's shape): cells hold one
        # point each, every point walks thousands of them
        _cluster("cluster_20kx16", 20_000, 16, 0.15, 26, 0.04, 0.04, 0.0),
        # two broad clusters: hundreds of iterations of a few moving points
        _cluster("cluster_250kx3", 250_000, 3, 0.03, 2, 0.05, 0.15, 0.05),
        # the largest run, from raw columns: normalise on the GPU, cluster,
        # keep labels and final positions on the device
        _cluster("cluster_1Mx3", 1_000_000, 3, 0.015, 50, 0.005, 0.03, 0.10, io="raw"),
        # the same loop started from the trained network's displacement
        _cluster("warm_500kx3", 500_000, 3, 0.02, 20, 0.005, 0.03, 0.10, io="warm"),
        # an eps sweep over several data sets of uneven size and dimension
        dict(name="sweep_6x8", kind="sweep", datasets=6, eps_count=8, n_min=1_000, n_max=100_000, sizes=4),
        # the eps search of full SynC: k-NN start, eps schedule, coding costs
        dict(name="search_100kx3", kind="search", n=100_000, d=3, k=5, candidates=16, clusters=20, std_lo=0.01,
             std_hi=0.04, noise=0.05),
        # brute-force SynC, the reference's second GPU entry point
        dict(name="simple_20kx2", kind="simple", n=20_000, d=2, eps=0.05, clusters=10, std_lo=0.02, std_hi=0.02,
             noise=0.05),
        # one update of every point, five dimensions, with neighbour counts
        dict(name="step_100kx5", kind="step", n=100_000, d=5, eps=0.05, clusters=20, std_lo=0.01, std_hi=0.04,
             noise=0.05),
        # an epoch of training the warm-start network (forward, backward, Adam)
        dict(name="train_65536", kind="train", rows=65_536, batch=2_048, epochs=1, d=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cluster"] * 6 + ["warm", "sweep", "search", "simple", "step", "train", "grad"])
    if kind in ("cluster", "warm"):
        d = 3 if kind == "warm" else rng.choice([2, 3, 3, 4, 5, 8, 14, 16])
        most = {2: 250_000, 3: 1_000_000, 4: 200_000, 5: 100_000}.get(d, 20_000)
        n = _log(rng, 150 if kind == "cluster" else 20_000, most)
        if d >= 8:
            eps = rng.uniform(0.05, 0.15)
        else:
            eps = rng.uniform(0.015, 0.03) if n > 100_000 else rng.uniform(0.02, 0.06)
        c = _cluster("", n, d, round(eps, 4), rng.randint(5, 50), 0.01, round(rng.uniform(0.02, 0.06), 3),
                     rng.choice([0.0, 0.05, 0.10]), io="warm" if kind == "warm" else
                     rng.choice(["device", "device", "dropin", "raw"]))
        if kind == "cluster" and c["io"] == "device" and n <= 50_000:
            c["stop"] = rng.choice(["flag", "flag", "lambda"])
        del c["name"]
        return c
    blobs = dict(clusters=rng.randint(5, 30), std_lo=0.01, std_hi=0.04, noise=0.05)
    if kind == "sweep":
        return dict(kind=kind, datasets=rng.randint(2, 8), eps_count=rng.choice([4, 8]), n_min=1_000,
                    n_max=_log(rng, 3_000, 60_000), sizes=rng.randrange(1 << 20))
    if kind == "search":
        return dict(kind=kind, n=_log(rng, 1_000, 80_000), d=rng.choice([2, 3]), k=rng.randint(2, 12),
                    candidates=rng.choice([8, 12, 16]), **blobs)
    if kind == "simple":
        return dict(kind=kind, n=_log(rng, 500, 20_000), d=rng.choice([2, 3, 5]), eps=round(rng.uniform(0.03, 0.06), 4),
                    **blobs)
    if kind == "step":
        d = rng.choice([2, 3, 5, 16])
        return dict(kind=kind, n=_log(rng, 1_000, 20_000 if d == 16 else 100_000), d=d,
                    eps=round(rng.uniform(0.1, 0.15) if d == 16 else rng.uniform(0.02, 0.06), 4), **blobs)
    if kind == "train":
        batch = rng.choice([512, 1_024, 2_048, 3_000])
        return dict(kind=kind, rows=batch * rng.randint(2, 24) + rng.randint(0, 511), batch=batch,
                    epochs=rng.randint(1, 2), d=rng.choice([2, 3, 3]))
    return dict(kind=kind, rows=_log(rng, 100, 65_536), d=rng.choice([1, 2, 3]))


def _points(case, seed, n=None, d=None):
    """n x d float32 host points in [0, 1]."""
    rng = np.random.default_rng(seed)
    n, d, k = n or case["n"], d or case["d"], case["clusters"]
    stds = rng.uniform(case["std_lo"], case["std_hi"], k)
    return data.blobs(rng, n, d, rng.uniform(0.1, 0.9, (k, d)), stds, np.ones(k), case["noise"])


def _raw_columns(X, seed):
    """The same points in the units a file would hold them in."""
    rng = np.random.default_rng(seed + 1)
    d = X.shape[1]
    return (X * rng.uniform(10, 200, d) + rng.uniform(-100, 100, d)).astype(F32)


def _training_rows(case, seed):
    """Feature rows and targets with the ranges of warm.features: offsets in
    [0, 1), then per neighbour cell log count, centroid and spread, zero where
    the cell is empty (about half of them), zero padding."""
    rng = np.random.default_rng(seed)
    m, d = case["rows"], case["d"]
    nb = 3 ** d
    full = (rng.random((m, nb, 1)) < 0.5).astype(F32)
    cells = np.concatenate([rng.random((m, nb, 1), F32), rng.random((m, nb, d), F32) * 2 - 1,
                            rng.random((m, nb, d), F32) * F32(0.4)], axis=2) * full
    width = (warm.feature_dim(d) + 15) // 16 * 16
    f = np.zeros((m, width), F32)
    f[:, :d] = rng.random((m, d), F32)
    f[:, d:warm.feature_dim(d)] = cells.reshape(m, -1)
    t = (f[:, d:2 * d] - F32(0.5) * f[:, :d] + F32(0.2) * rng.standard_normal((m, d)).astype(F32)).astype(F32)
    return f, np.ascontiguousarray(t)


def _sweep_sizes(case):
    rng = random.Random(case["sizes"])
    return [(_log(rng, case["n_min"], case["n_max"]), rng.choice([2, 3, 5]), rng.randint(5, 30))
            for _ in range(case["datasets"])]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "seed": seed}
    if kind in ("train", "grad"):
        s["feats"], s["targets"] = _training_rows(case, seed)
        s["model"] = warm.Model(case["d"], seed=seed)
        return s
    if kind == "sweep":
        eps = np.logspace(np.log10(0.01), np.log10(0.08), case["eps_count"]).astype(F32)
        s["instances"], s["labels"] = [], []
        for k, (n, d, clusters) in enumerate(_sweep_sizes(case)):
            c = dict(n=n, d=d, clusters=clusters, std_lo=0.01, std_hi=0.04, noise=0.05)
            X = torch.from_numpy(_points(c, 1000 * seed + k)).cuda()
            for e in eps:
                s["instances"].append((X, float(e)))
                s["labels"].append(torch.empty(n, dtype=torch.int32, device="cuda"))
        return s
    X = _points(case, seed)
    if case.get("io") == "dropin":
        s["X"] = torch.from_numpy(X)
        return s
    if case.get("io") == "raw":
        X = _raw_columns(X, seed)
    s["X"] = torch.from_numpy(X).cuda()
    if kind in ("cluster", "search"):
        s["labels"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
    if case.get("io") in ("raw", "warm"):
        s["positions"] = torch.empty_like(s["X"])
        s["normalised"] = torch.empty_like(s["X"])
    if case.get("io") == "warm":
        s["model"] = warm.default_model(3)
    return s


def _counts(info):
    return [info["iterations"], info["n_clusters"]]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "cluster":
        if case["io"] == "dropin":
            C, _, _, _ = eggsync.EGG_SynC(s["X"], case["eps"])
            return {"labels": C}
        if case["io"] == "raw":
            X, lo, hi = eggsync.normalize(s["X"], out=s["normalised"])
            lab, info = eggsync.egg_sync(X, case["eps"], labels_out=s["labels"], positions_out=s["positions"])
            return {"labels": lab, "counts": _counts(info), "positions": s["positions"], "x": X, "lo": lo, "hi": hi}
        if case["io"] == "warm":
            lab, info = eggsync.egg_sync(s["X"], case["eps"], labels_out=s["labels"], positions_out=s["positions"],
                                         warm_start=s["model"])
            return {"labels": lab, "counts": _counts(info), "positions": s["positions"]}
        lab, info = eggsync.egg_sync(s["X"], case["eps"], LAMBDA, stop_rule=case["stop"], labels_out=s["labels"])
        return {"labels": lab, "counts": _counts(info)}
    if kind == "sweep":
        res, _ = eggsync.egg_sync_batch(s["instances"], labels_out=s["labels"])
        return {"labels": torch.cat([lab for lab, _ in res]), "counts": np.array([_counts(i) for _, i in res])}
    if kind == "search":
        lab, info = eggsync.mdl_search(s["X"], case["k"], max_candidates=case["candidates"], labels_out=s["labels"])
        return {"labels": lab, "nn": [info["eps0"], info["eps1"]], "eps": np.array(info["eps"], F32),
                "costs": np.array(info["costs"]), "clusters": np.array(info["clusters"]), "best": info["best"]}
    if kind == "simple":
        P = np.empty((case["n"], case["d"]), F32)
        lab, info = eggsync.simple_sync(s["X"], case["eps"], LAMBDA, positions_out=P)
        return {"labels": lab, "positions": P, "iterations": info["iterations"]}
    if kind == "step":
        x, cnt, flags = eggsync.egg_step(s["X"], case["eps"])
        return {"x": x, "counts": cnt, "flags": list(flags)}
    if kind == "grad":
        loss, g = warm.grad(s["model"], s["feats"], s["targets"])
        return {"loss": loss, "grads": g}
    model = s["model"].copy()
    losses = warm.train(model, s["feats"], s["targets"], epochs=case["epochs"], batch=case["batch"], lr=2e-3,
                        seed=s["seed"])
    return {"losses": losses, "weights": model.w}


def work(case):
    """Inputs read once, outputs written once; operations only where their
    number is given by the sizes (the pairs of the brute-force path, the
    network's products)."""
    kind = case["kind"]
    if kind in ("train", "grad"):
        d, h = case["d"], warm.HIDDEN
        f = warm.feature_dim(d)
        rows = case["rows"] if kind == "grad" else case["rows"] // case["batch"] * case["batch"] * case["epochs"]
        params = f * h + h * h + h * d + 2 * h + d
        # forward, weight gradients, input gradients of layers 2 and 3
        flops = rows * (4 * (f * h + h * h + h * d) + 2 * (h * h + h * d))
        return {"bytes": 4 * case["rows"] * (f + d) + 8 * params, "flops": flops}
    if kind == "sweep":
        sizes = _sweep_sizes(case)
        return {"bytes": sum(4 * n * d + 4 * n * case["eps_count"] for n, d, _ in sizes), "flops": 0}
    n, d = case["n"], case["d"]
    w = {"bytes": 4 * n * d + 4 * n, "flops": 0}
    if case.get("io") == "raw":
        w["bytes"] += 8 * n * d  # normalised points, final positions
    elif case.get("io") == "warm":
        w["bytes"] += 4 * n * d
        f, h = warm.feature_dim(3), warm.HIDDEN
        w["flops"] = 2 * n * (f * h + h * h + h * d)
    elif kind == "step":
        w["bytes"] += 4 * n * d
    elif kind == "simple":
        w["bytes"] += 4 * n * d
        w["flops"] = n * n * 3 * d
    return w


def _knn64(X, k):
    n = len(X)
    sums = torch.zeros(2, dtype=torch.float64, device="cuda")
    rows = max(1, int(1e8) // n)
    for b in range(0, n, rows):
        d2 = torch.zeros(min(rows, n - b), n, dtype=torch.float64, device="cuda")
        for c in range(X.shape[1]):
            d2 += (X[b:b + rows, c, None] - X[None, :, c]) ** 2
        v = d2.topk(k + 2, dim=1, largest=False, sorted=True).values  # the first is the point itself
        sums += v[:, k:k + 2].sqrt().sum(0)
    return [float(v) / n for v in sums]


def _simple64(X, eps):
    """Brute-force SynC: 64-bit sums, neighbourhoods of the float32 positions."""
    x = X.double()
    n, it, r = len(x), 0, 0.0
    rows = max(1, int(5e7) // n)
    while r < float(F32(LAMBDA)) and it < 100:
        out, r = torch.empty_like(x), 0.0
        for b in range(0, n, rows):
            diff = x[None] - x[b:b + rows, None]
            dist = diff.square().sum(2).sqrt()
            near = dist.float() <= F32(eps)
            cnt = near.sum(1)
            out[b:b + rows] = x[b:b + rows] + (diff.sin() * near[..., None]).sum(1) / cnt[:, None]
            r += float(((-dist).exp() * near).sum(1).div(cnt).sum())
        x, r, it = out.float().double(), r / n, it + 1
    return x


def _step64(X, eps):
    """One EGG-SynC update in 64 bits.  The neighbourhood is the reference's:
    the points within eps that lie in a cell passing its box test (the sum
    over the dimensions of the squared distance to the nearer face)."""
    n, d = X.shape
    eps = float(F32(eps))
    side = float(F32(math.sqrt((eps / 2) ** 2 / d)))
    width = int(F32(1.0) / F32(side))
    cell = (X / F32(side)).int().clamp(0, width - 1)
    out = torch.empty(n, d, dtype=torch.float64, device="cuda")
    rows = max(1, int(4e7) // n)
    for b in range(0, n, rows):
        box = torch.zeros(min(rows, n - b), n, device="cuda")
        d2 = torch.zeros_like(box)
        for c in range(d):
            x = X[b:b + rows, c, None].double()
            face = [((cell[None, :, c].double() + k) * side - x).float().square() for k in (0, 1)]
            box += torch.minimum(*face)
            d2 += (X[None, :, c] - X[b:b + rows, c, None]).square()
        near = (box.sqrt() <= eps) & (d2.sqrt() <= eps)
        cnt = near.sum(1)
        for c in range(d):
            x = X[b:b + rows, c].double()
            s = ((X[None, :, c].double() - x[:, None]).sin() * near).sum(1)
            out[b:b + rows, c] = x + s / cnt
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        f, t = (torch.from_numpy(a).cuda().double() for a in _training_rows(case, seed))
        w = {k: torch.from_numpy(v).cuda().double().requires_grad_() for k, v in warm.Model(case["d"], seed=seed).w.items()}
        h = (f[:, :warm.feature_dim(case["d"])] @ w["w1"] + w["b1"]).relu()
        y = (h @ w["w2"] + w["b2"]).relu() @ w["w3"] + w["b3"]
        loss = (y - t).square().mean()
        loss.backward()
        return {"loss": float(loss.detach()), "grads": {k: v.grad for k, v in w.items()}}
    if kind not in ("cluster", "search", "simple", "step"):
        return None  # labels of a batch; weights after a shuffled epoch
    X = _points(case, seed)
    if kind == "cluster":
        if case["io"] != "raw":
            return None  # labels; positions decided by thresholds in every iteration
        x = torch.from_numpy(_raw_columns(X, seed)).double()
        lo, hi = x.min(0).values, x.max(0).values
        return {"labels": None, "counts": None, "positions": None, "x": (x - lo) / (hi - lo), "lo": lo, "hi": hi}
    X = torch.from_numpy(X).cuda()
    if kind == "search":
        nn = _knn64(X.double(), case["k"])
        return {"labels": None, "nn": nn, "eps": None, "costs": None, "clusters": None, "best": None}
    if kind == "simple":
        return {"labels": None, "positions": _simple64(X, case["eps"]), "iterations": None}
    return {"x": _step64(X, case["eps"]), "counts": None, "flags": None}
