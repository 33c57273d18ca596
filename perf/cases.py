"""The work that users of this framework have it do, as measurable cases.

Each case is one call (or one training step) through a public entry point, at
sizes taken from the benchmark configurations and the tests, or generic ones,
odd sizes among them.  ``listed()`` names the standing cases, ``draw(rng)``
makes another of the same ranges, ``prepare`` builds what a program holds
before the call, ``run`` is one pass, ``work`` counts what a pass cannot do
without and ``exact`` gives the float64 values of its outputs.
"""
import math
import warnings

import numpy as np
import torch

from mlxlearn_b200.autograd import chamfer_loss_batch, knn_distances
from mlxlearn_b200.batch import KnnBatch
from mlxlearn_b200.index import NeighborIndex
from mlxlearn_b200.neighbors import (KNeighborsClassifier, RadiusNeighborsClassifier,
                                     RadiusNeighborsRegressor)

DEVICE = "cuda"


def listed():
    return [
        # one query against a small index: an online lookup, bound by latency
        {"name": "query_one_10000x64", "kind": "query", "data": "normal", "n": 10_000, "d": 64,
         "m": 1, "k": 5},
        # a small table searched once, the ordinary interactive call
        {"name": "query_10000x64_2000q", "kind": "query", "data": "normal", "n": 10_000, "d": 64,
         "m": 2_000, "k": 5},
        # the headline: a large embedding table and a large batch
        {"name": "query_1Mx128_100kq", "kind": "query", "data": "mixture", "n": 1_000_000,
         "d": 128, "m": 100_000, "k": 10},
        # images scaled to [0, 1] (not integers any more): wide float rows
        {"name": "query_60000x784_10000q", "kind": "query", "data": "pixels01", "n": 60_000,
         "d": 784, "m": 10_000, "k": 5},
        # geographic or tabular points, few columns
        {"name": "query_200003x8_50021q", "kind": "query", "data": "normal", "n": 200_003, "d": 8,
         "m": 50_021, "k": 5},
        # the neighbour graph of an embedding (t-SNE, UMAP): every row against the others, large k
        {"name": "graph_60013x100_k50", "kind": "graph", "data": "mixture", "n": 60_013, "d": 100,
         "k": 50},
        # classification of 8-bit images, host arrays in and probabilities out
        {"name": "classify_60000x784_10000q", "kind": "classify", "n": 60_000, "d": 784,
         "m": 10_000, "k": 5, "classes": 10},
        # fixed-radius regression weighted by distance: neighbourhoods with their distances
        {"name": "radius_regress_100003x24_30011q", "kind": "radius_regress", "n": 100_003,
         "d": 24, "m": 30_011, "near": 50},
        # fixed-radius classification, host arrays in and probabilities out
        {"name": "radius_classify_200000x32_50000q", "kind": "radius_classify", "n": 200_000,
         "d": 32, "m": 50_000, "near": 50},
        # many tenants' indexes of uneven size answered by one planned run
        {"name": "batch_32_uneven", "kind": "batch", "problems": 32, "layout": 5},
        # a training step of a point-cloud model: Chamfer loss, forward and backward
        {"name": "chamfer_64x8192x3", "kind": "chamfer", "pairs": 64, "points": 8_192},
        # a training step on embeddings: distances to the k nearest others, forward and backward
        {"name": "self_grad_32768x64_k8", "kind": "self_grad", "n": 32_768, "d": 64, "k": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query"] * 5 + ["graph", "classify", "radius_regress",
                                       "radius_classify", "batch", "chamfer", "self_grad"])
    if kind == "query":
        data = rng.choice(["normal", "mixture", "pixels01"])
        n, m = _log_int(rng, 5_000, 1_000_000), _log_int(rng, 1, 100_000)
        d = _log_int(rng, 3, 256) if data != "pixels01" else rng.randint(196, 960)
        if d > 128:
            n = min(n, 128_000_000 // d)
        return {"kind": kind, "data": data, "n": n, "d": d, "m": m,
                "k": rng.choice([1, 3, 5, 8, 10, 15, 20, 32, 50])}
    if kind == "graph":
        return {"kind": kind, "data": rng.choice(["normal", "mixture"]),
                "n": _log_int(rng, 5_000, 80_000), "d": _log_int(rng, 16, 200),
                "k": rng.choice([5, 10, 15, 30, 50])}
    if kind == "classify":
        return {"kind": kind, "n": _log_int(rng, 5_000, 60_000), "d": rng.randint(64, 784),
                "m": _log_int(rng, 100, 10_000), "k": rng.choice([1, 3, 5, 9, 15]),
                "classes": rng.choice([2, 10, 47])}
    if kind in ("radius_regress", "radius_classify"):
        return {"kind": kind, "n": _log_int(rng, 10_000, 200_000), "d": rng.randint(8, 64),
                "m": _log_int(rng, 500, 50_000), "near": rng.choice([5, 20, 50, 100])}
    if kind == "batch":
        return {"kind": kind, "problems": rng.randint(8, 32), "layout": rng.randrange(1 << 20)}
    if kind == "chamfer":
        return {"kind": kind, "pairs": rng.randint(1, 64), "points": _log_int(rng, 500, 8_192)}
    return {"kind": kind, "n": _log_int(rng, 2_000, 65_536), "d": _log_int(rng, 16, 128),
            "k": rng.choice([4, 8, 15])}


# ------------------------------------------------------------------- inputs
def _generator(seed, stream):
    return torch.Generator(device=DEVICE).manual_seed((int(seed) * 64 + stream) % (1 << 62))


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device=DEVICE)


def _mixture(g, rows, centres, sigma):
    label = torch.randint(len(centres), (rows,), generator=g, device=DEVICE)
    return centres[label] + sigma * _normal(g, rows, centres.shape[1]), label


def _pixels(g, rows, templates):
    """Integer pixels 0..255 as float32, about 80% zeros, around class templates."""
    label = torch.randint(len(templates), (rows,), generator=g, device=DEVICE)
    out = torch.empty((rows, templates.shape[1]), device=DEVICE)
    for a in range(0, rows, 8_192):
        t = templates[label[a:a + 8_192]]
        mask = t ^ (torch.rand(t.shape, generator=g, device=DEVICE) < 0.03)
        out[a:a + 8_192] = torch.randint(1, 256, t.shape, generator=g, device=DEVICE) * mask
    return out, label


def _rows(case, seed):
    """Training rows and queries of a search case (float32, on the GPU)."""
    n, d, m, data = case["n"], case["d"], case.get("m", 0), case["data"]
    gx, gq, gc = _generator(seed, 0), _generator(seed, 1), _generator(seed, 2)
    if data == "normal":
        return _normal(gx, n, d), _normal(gq, m, d)
    if data == "mixture":
        centres = 2 * torch.rand((1_024, d), generator=gc, device=DEVICE) - 1
        return _mixture(gx, n, centres, 0.1)[0], _mixture(gq, m, centres, 0.1)[0]
    templates = torch.rand((10, d), generator=gc, device=DEVICE) < 0.2
    return _pixels(gx, n, templates)[0] / 255, _pixels(gq, m, templates)[0] / 255


def _images(case, seed):
    templates = torch.rand((case["classes"], case["d"]), generator=_generator(seed, 2),
                           device=DEVICE) < 0.2
    X, y = _pixels(_generator(seed, 0), case["n"], templates)
    Q, _ = _pixels(_generator(seed, 1), case["m"], templates)
    return X, y, Q


def _radius_rows(case, seed):
    """Ten classes N(c, I), c ~ N(0, 4 I), with the class (classification) or a
    smooth float64 target (regression) of each training row; the radius gives a
    median of about `near` neighbours a query."""
    centres = 2 * _normal(_generator(seed, 2), 10, case["d"])
    X, y = _mixture(_generator(seed, 0), case["n"], centres, 1.0)
    Q, _ = _mixture(_generator(seed, 1), case["m"], centres, 1.0)
    d2 = _squared(Q[:256].double(), X.double())
    near = torch.kthvalue(d2, min(case["near"], case["n"]), dim=1).values
    if case["kind"] == "radius_regress":
        y = X[:, :8].double().sin().sum(1) + y
    return X, y, Q, math.sqrt(max(float(near.median()), 0.0))


def _problems(case):
    """(n, m, d, k) of each problem of a batch."""
    rng = np.random.default_rng(case["layout"])
    out = []
    for _ in range(case["problems"]):
        n = int(round(math.exp(rng.uniform(math.log(1_000), math.log(200_000)))))
        m = int(round(math.exp(rng.uniform(math.log(100), math.log(20_000)))))
        out.append((n, m, int(rng.choice((16, 32, 64, 128, 256))), int(rng.choice((1, 5, 10, 50)))))
    return out


def _batch_rows(case, seed):
    """Rows N(0, 1), 1% of each problem's training rows duplicated."""
    g = _generator(seed, 0)
    out = []
    for n, m, d, k in _problems(case):
        X = _normal(g, n, d)
        dup = max(1, n // 100)
        order = torch.randperm(n, generator=g, device=DEVICE)
        X[order[:dup]] = X[order[-dup:]]
        out.append((X, _normal(g, m, d), k))
    return out


def _clouds(case, seed):
    """Two sets of clouds [pairs, points, 3] on the unit sphere, jitter 0.01."""
    g = _generator(seed, 0)
    out = []
    for _ in range(2):
        v = _normal(g, case["pairs"], case["points"], 3)
        out.append(v / v.norm(dim=2, keepdim=True) + 0.01 * _normal(g, *v.shape))
    return out


# ------------------------------------------------------------------- passes
def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind in ("query", "graph"):
        X, Q = _rows(case, seed)
        state["index"] = NeighborIndex.from_device(X)
        state["Q"] = Q if kind == "query" else X
    elif kind == "classify":
        X, y, Q = _images(case, seed)
        state["model"] = KNeighborsClassifier(n_neighbors=case["k"]).fit(X.cpu().numpy(),
                                                                        y.cpu().numpy())
        state["Q"] = Q.cpu().numpy()
    elif kind in ("radius_regress", "radius_classify"):
        X, y, Q, radius = _radius_rows(case, seed)
        model = (RadiusNeighborsRegressor(radius=radius, weights="distance")
                 if kind == "radius_regress" else
                 RadiusNeighborsClassifier(radius=radius, outlier_label="most_frequent"))
        state["model"] = model.fit(X.cpu().numpy(), y.cpu().numpy())
        state["Q"] = Q.cpu().numpy()
    elif kind == "batch":
        state["batch"] = KnnBatch([(NeighborIndex.from_device(X), Q, k)
                                   for X, Q, k in _batch_rows(case, seed)])
    elif kind == "chamfer":
        state["A"], state["B"] = (c.requires_grad_() for c in _clouds(case, seed))
    else:
        state["E"] = _normal(_generator(seed, 0), case["n"], case["d"]).requires_grad_()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("query", "graph"):
        return state["index"].query_device(state["Q"], case["k"], exclude_self=kind == "graph")
    if kind in ("classify", "radius_classify"):
        return state["model"].predict_proba(state["Q"])
    if kind == "radius_regress":
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")  # queries without a neighbour predict NaN
            return state["model"].predict(state["Q"])
    if kind == "batch":
        return state["batch"]()
    if kind == "chamfer":
        loss = chamfer_loss_batch(state["A"], state["B"])
        return (loss.detach(), *torch.autograd.grad(loss, (state["A"], state["B"])))
    dist, idx = knn_distances(state["E"], None, case["k"])
    grad, = torch.autograd.grad(dist.mean(), (state["E"],))
    return dist.detach(), idx, grad


def work(case):
    """One pass: two operations per coordinate of every (query, row) pair; the
    rows and queries read once as float32 and the outputs written once."""
    kind = case["kind"]
    if kind in ("query", "graph"):
        n, d, k = case["n"], case["d"], case["k"]
        m = case["m"] if kind == "query" else n
        return {"flops": 2 * n * m * d, "bytes": 4 * n * d + (4 * m * d if m != n else 0)
                + 16 * m * k}
    if kind == "classify":
        n, d, m = case["n"], case["d"], case["m"]
        return {"flops": 2 * n * m * d, "bytes": 4 * d * (n + m) + 8 * m * case["classes"]}
    if kind in ("radius_regress", "radius_classify"):
        n, d, m = case["n"], case["d"], case["m"]
        return {"flops": 2 * n * m * d,
                "bytes": 4 * d * (n + m) + (8 if kind == "radius_regress" else 80) * m}
    if kind == "batch":
        ps = _problems(case)
        return {"flops": sum(2 * n * m * d for n, m, d, _ in ps),
                "bytes": sum(4 * d * (n + m) + 16 * m * k for n, m, d, k in ps)}
    if kind == "chamfer":
        p, c = case["points"], case["pairs"]
        return {"flops": 2 * c * p * p * 8, "bytes": 2 * c * p * 3 * 8 + 4}
    n, d, k = case["n"], case["d"], case["k"]
    return {"flops": 2 * n * n * d, "bytes": 8 * n * d + 12 * n * k}


# ------------------------------------------------------------- exact values
def _squared(Q, X):
    """Squared distances of float64 rows by inner products (about 1e-13)."""
    return ((Q * Q).sum(1, keepdim=True) + (X * X).sum(1)).addmm_(Q, X.t(), alpha=-2)


def _exact_nearest(X, Q, k, exclude_self=False):
    """float64 squared distances [m, k] and rows of the k nearest: candidates
    by inner products on centred rows, then direct differences."""
    c = X.double().mean(0)
    Xd, Qd = X.double() - c, Q.double() - c
    keep = min(k + 8 + exclude_self, len(X))
    step = max(1, min(len(Q), (1 << 29) // len(X)))
    dist, rows = [], []
    for a in range(0, len(Q), step):
        q = Qd[a:a + step]
        d2 = _squared(q, Xd)
        if exclude_self:
            i = torch.arange(len(q), device=q.device)
            d2[i, a + i] = math.inf
        cand = d2.topk(keep, largest=False, sorted=False).indices.sort(dim=1).values
        del d2
        part = max(1, (1 << 27) // (keep * X.shape[1]))
        for b in range(0, len(q), part):
            cb = cand[b:b + part]
            s = (Q[a + b:a + b + len(cb)].double()[:, None] - X[cb].double()).square().sum(2)
            if exclude_self:
                self_row = torch.arange(a + b, a + b + len(cb), device=s.device)
                s.masked_fill_(cb == self_row[:, None], math.inf)
            s, order = s.sort(dim=1, stable=True)
            dist.append(s[:, :k])
            rows.append(cb.gather(1, order[:, :k]))
    return torch.cat(dist), torch.cat(rows)


def exact(case, seed):
    """What `run` returns, from float64 arithmetic; None for whole numbers."""
    kind = case["kind"]
    if kind in ("query", "graph"):
        X, Q = _rows(case, seed)
        d2, _ = _exact_nearest(X, Q if kind == "query" else X, case["k"], kind == "graph")
        return d2.sqrt(), None
    if kind == "classify":
        X, y, Q = _images(case, seed)
        Xd, key = X.double(), torch.arange(case["n"], device=DEVICE, dtype=torch.float64)
        votes = torch.zeros((case["m"], case["classes"]), device=DEVICE, dtype=torch.float64)
        for a in range(0, case["m"], 2_048):
            # integer data: the squared distances are exact, ties go to the smaller row
            s = _squared(Q[a:a + 2_048].double(), Xd) * float(1 << 17) + key
            near = y[s.topk(case["k"], largest=False).indices]
            votes[a:a + 2_048].scatter_add_(1, near, torch.ones_like(near, dtype=torch.float64))
        present = torch.bincount(y, minlength=case["classes"]) > 0
        return (votes[:, present] / case["k"]).cpu().numpy()
    if kind in ("radius_regress", "radius_classify"):
        X, y, Q, radius = _radius_rows(case, seed)
        c = X.double().mean(0)
        Xd, Qd = X.double() - c, Q.double() - c
        limit = radius * radius
        step = max(1, (1 << 29) // len(X))
        out = []
        for a in range(0, len(Q), step):
            near = _squared(Qd[a:a + step], Xd) <= limit * (1 + 1e-9)
            r, col = near.nonzero(as_tuple=True)
            rows = len(near)
            del near
            s = torch.empty(len(r), device=DEVICE, dtype=torch.float64)
            for b in range(0, len(r), 1 << 22):
                e = b + (1 << 22)
                s[b:e] = (Q[a + r[b:e]].double() - X[col[b:e]].double()).square().sum(1)
            inside = s <= limit
            r, col, s = r[inside], col[inside], s[inside]
            if kind == "radius_classify":
                out.append(torch.bincount(r * 10 + y[col], minlength=rows * 10).view(rows, 10))
                continue
            sums = torch.zeros((2, rows), device=DEVICE, dtype=torch.float64)
            sums[0].index_add_(0, r, y[col] / s.sqrt())
            sums[1].index_add_(0, r, 1 / s.sqrt())
            out.append(sums[0] / sums[1])
        out = torch.cat(out)
        if kind == "radius_regress":
            return out.cpu().numpy()
        votes, counts = out.double(), torch.bincount(y, minlength=10)
        votes[votes.sum(1) == 0, counts.argmax()] = 1.0
        votes = votes[:, counts > 0]
        return (votes / votes.sum(1, keepdim=True)).cpu().numpy()
    if kind == "batch":
        return [(_exact_nearest(X, Q, k)[0].sqrt(), None) for X, Q, k in _batch_rows(case, seed)]
    if kind == "chamfer":
        A, B = _clouds(case, seed)
        total = torch.zeros((), device=DEVICE, dtype=torch.float64)
        grads = [torch.zeros(A.shape, device=DEVICE, dtype=torch.float64) for _ in range(2)]
        for p in range(case["pairs"]):
            for x, y, gx, gy in ((A[p], B[p], grads[0][p], grads[1][p]),
                                 (B[p], A[p], grads[1][p], grads[0][p])):
                d2, rows = _exact_nearest(y, x, 1)
                g = 2 * (x.double() - y[rows[:, 0]].double())
                total += d2.sum()
                gx += g
                gy.index_add_(0, rows[:, 0], -g)
        return (total, *grads)
    E = _normal(_generator(seed, 0), case["n"], case["d"])
    k = case["k"]
    d2, rows = _exact_nearest(E, E, k, True)
    dist = d2.sqrt()
    grad = torch.zeros(E.shape, device=DEVICE, dtype=torch.float64)
    for j in range(k):
        g = (E.double() - E[rows[:, j]].double()) / dist[:, j:j + 1] / dist.numel()
        grad += g
        grad.index_add_(0, rows[:, j], -g)
    return dist, None, grad
