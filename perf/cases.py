"""Workloads that the distance path is timed on.

Every case is one call (or one training step) that a program makes through the
public entry points of ``wildboar_gb300.distance``: distance matrices of the
elastic metrics, nearest neighbours, shapelet scans, the batched float32 form
and the differentiable form.  ``listed`` gives fixed sizes, ``draw`` others of
the same ranges; ``exact`` restates every result in float64 with plain torch
and numpy (anti-diagonal sweeps over all pairs at once).

Series are the repository's benchmark data: seeded Gaussian random walks
(z-normalised fragments for shapelets, noisy prototypes for the barycenter
step).
"""

import math

import numpy as np
import torch

from wildboar_gb300.distance import (
    argmin_distance,
    pairwise_distance,
    pairwise_subsequence_distance,
)
from wildboar_gb300.distance.autograd import dtw_matrix, soft_assignment_loss
from wildboar_gb300.distance.batched import BatchedDTW

# the elastic metrics by the shape of their recurrence: dtw and its relatives
# run with the band that users set, the edit distances with the default full
# band
WARPING = ("dtw", "ddtw", "wdtw", "adtw")
EDIT = ("lcss", "edr", "erp", "msm", "twe")


def listed():
    return [
        # a first look at a small data set from numpy: the latency of one call
        dict(name="pairwise_small_host", family="pairwise", metric="dtw", r=0.1,
             nx=100, ny=100, lx=128, ly=128, host=True),
        # the distance matrix of a classification or clustering study: a
        # Sakoe-Chiba band of a tenth of the length
        dict(name="pairwise_dtw", family="pairwise", metric="dtw", r=0.1,
             nx=1000, ny=1000, lx=512, ly=512, host=False),
        # two collections of different lengths without a band restriction
        # (r = 1 is the default)
        dict(name="pairwise_dtw_full_band", family="pairwise", metric="dtw", r=1.0,
             nx=310, ny=301, lx=400, ly=361, host=False),
        # weighted dtw with its default parameters, from numpy
        dict(name="pairwise_wdtw_host", family="pairwise", metric="wdtw", r=1.0,
             nx=500, ny=403, lx=256, ly=256, host=True),
        # edit distance on real sequences
        dict(name="pairwise_edr", family="edit", metric="edr", nx=500, ny=500, lx=256,
             ly=256),
        # move-split-merge
        dict(name="pairwise_msm", family="edit", metric="msm", nx=301, ny=290, lx=256,
             ly=250),
        # the default metric of every entry point
        dict(name="pairwise_euclidean", family="euclidean", nx=2000, ny=1500, length=700),
        # k-nearest-neighbour search under dtw
        dict(name="argmin_knn", family="argmin", r=0.1, nx=500, ny=2000, length=512, k=5),
        # the attribute matrix of a shapelet transform (z-normalised windows)
        dict(name="subsequence_scaled", family="subsequence", metric="scaled_euclidean", r=1.0,
             m=2000, n=400, length=1024, low=16, high=128),
        # shapelets compared under dtw
        dict(name="subsequence_dtw", family="subsequence", metric="dtw", r=0.1, m=200, n=100,
             length=1024, low=16, high=128),
        # a ragged multivariate float32 batch on kept buffers, graph replayed
        dict(name="batched_ragged", family="batched", r=0.1, n=4096, dims=3, low=32,
             high=2048),
        # forward and backward of a dtw-barycenter step
        dict(name="barycenter_step", family="gradient", r=0.2, nx=4096, ny=32, length=256),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    largest = {}
    for c in listed():
        w = work(c)["flops"]
        largest[c["family"]] = max(largest.get(c["family"], 0.0), w)
    family = rng.choice(["pairwise", "pairwise", "edit", "edit", "euclidean", "argmin",
                         "subsequence", "subsequence", "batched", "gradient"])
    while True:
        if family == "pairwise":
            lx = _log_int(rng, 24, 1024)
            case = dict(family=family, metric=rng.choice(WARPING),
                        r=rng.choice([0.05, 0.1, 0.2, 0.5, 1.0]),
                        nx=_log_int(rng, 4, 2000), ny=_log_int(rng, 4, 2000), lx=lx,
                        ly=lx if rng.random() < 0.6 else _log_int(rng, 24, 1024),
                        host=rng.random() < 0.4)
        elif family == "edit":
            lx = _log_int(rng, 24, 512)
            case = dict(family=family, metric=rng.choice(EDIT), nx=_log_int(rng, 4, 1000),
                        ny=_log_int(rng, 4, 1000), lx=lx,
                        ly=lx if rng.random() < 0.6 else _log_int(rng, 24, 512))
        elif family == "euclidean":
            case = dict(family=family, nx=_log_int(rng, 16, 4000), ny=_log_int(rng, 16, 4000),
                        length=_log_int(rng, 16, 2048))
        elif family == "argmin":
            case = dict(family=family, r=rng.choice([0.05, 0.1, 0.2, 1.0]),
                        nx=_log_int(rng, 10, 1000), ny=_log_int(rng, 100, 4000),
                        length=_log_int(rng, 32, 512), k=rng.choice([1, 3, 5, 10]))
        elif family == "subsequence":
            metric = rng.choice(["euclidean", "scaled_euclidean", "dtw"])
            low = rng.randint(8, 24)
            case = dict(family=family, metric=metric, r=rng.choice([0.1, 0.2]),
                        m=_log_int(rng, 20, 2000), n=_log_int(rng, 20, 400),
                        length=_log_int(rng, 200, 1024), low=low,
                        high=rng.randint(low + 8, 128))
        elif family == "batched":
            high = _log_int(rng, 128, 2048)
            case = dict(family=family, r=rng.choice([0.05, 0.1, 0.2]), n=_log_int(rng, 256, 8192),
                        dims=rng.choice([1, 2, 3]), low=max(16, high // 64), high=high)
        else:
            case = dict(family=family, r=rng.choice([0.1, 0.2, 0.5]), nx=_log_int(rng, 128, 4096),
                        ny=_log_int(rng, 2, 64), length=_log_int(rng, 48, 512))
        # between a thousandth of the family's largest listed case and all of it
        if largest[family] * 1e-3 <= work(case)["flops"] <= largest[family]:
            return case


# --------------------------------------------------------------------------
# inputs


def _walks(rng, n, length):
    return np.cumsum(rng.standard_normal((n, length)), axis=1)


def _shapelets(rng, m, low, high):
    out = []
    for length in rng.integers(low, high + 1, size=m):
        s = np.cumsum(rng.standard_normal(int(length)))
        out.append((s - s.mean()) / (s.std() + 1e-12))
    return out


def _arrays(case, seed):
    """The host arrays of a case: what ``prepare`` uploads and ``exact`` reads."""
    rng = np.random.default_rng(seed)
    f = case["family"]
    if f in ("pairwise", "edit"):
        return _walks(rng, case["nx"], case["lx"]), _walks(rng, case["ny"], case["ly"])
    if f in ("euclidean", "argmin"):
        return (_walks(rng, case["nx"], case["length"]),
                _walks(rng, case["ny"], case["length"]))
    if f == "subsequence":
        return (_shapelets(rng, case["m"], case["low"], case["high"]),
                _walks(rng, case["n"], case["length"]))
    if f == "batched":
        out = []
        for _ in range(2):
            a = np.cumsum(rng.standard_normal((case["n"], case["dims"], case["high"])),
                          axis=2).astype(np.float32)
            lens = rng.integers(case["low"], case["high"] + 1, size=case["n"])
            pad = np.arange(case["high"])[None, None, :] >= lens[:, None, None]
            a[np.broadcast_to(pad, a.shape)] = np.nan
            out.append(a)
        return tuple(out)
    # prototypes (sines and random walks) plus noise, and perturbed centroids
    t = np.arange(case["length"])
    k = case["ny"]
    protos = np.stack([np.sin(2 * np.pi * (1 + i % 7) * t / case["length"] + i)
                       if i % 2 == 0
                       else np.cumsum(rng.standard_normal(case["length"])) / 8.0
                       for i in range(k)])
    x = protos[rng.integers(0, k, size=case["nx"])]
    x = x + 0.1 * rng.standard_normal(x.shape)
    c = protos + 0.1 * rng.standard_normal(protos.shape)
    return x.astype(np.float32), c.astype(np.float32)


def _params(case):
    f = case["family"]
    if f == "pairwise" or f == "argmin":
        return {"r": case["r"]}
    if f == "edit":
        # a tenth of the data's spread for the metrics with a tolerance; the
        # other parameters at their defaults
        return {"epsilon": 1.6} if case["metric"] in ("lcss", "edr") else {}
    if f == "subsequence":
        return {"r": case["r"]} if case["metric"] == "dtw" else {}
    return {}


def prepare(case, seed):
    a, b = _arrays(case, seed)
    f = case["family"]
    state = {"case": case, "params": _params(case)}
    if f == "subsequence":
        state["y"] = a
        state["x"] = torch.as_tensor(b, device="cuda")
    elif case.get("host"):
        state["x"], state["y"] = a, b
    else:
        state["x"] = torch.as_tensor(a, device="cuda")
        state["y"] = torch.as_tensor(b, device="cuda")
    if f == "batched":
        state["handle"] = BatchedDTW(state["x"], state["y"], case["r"], tune=False)
    if f == "gradient":
        state["x"].requires_grad_(True)
        state["y"].requires_grad_(True)
    return state


def run(state):
    case, x, y = state["case"], state["x"], state["y"]
    f = case["family"]
    if f in ("pairwise", "edit"):
        return pairwise_distance(x, y, metric=case["metric"], metric_params=state["params"])
    if f == "euclidean":
        return pairwise_distance(x, y)
    if f == "argmin":
        indices, distances = argmin_distance(x, y, k=case["k"], metric="dtw",
                                             metric_params=state["params"], sorted=True,
                                             return_distance=True)
        return {"indices": indices, "distances": distances}
    if f == "subsequence":
        distances, indices = pairwise_subsequence_distance(
            y, x, metric=case["metric"], metric_params=state["params"], return_index=True)
        return {"distances": distances, "indices": indices}
    if f == "batched":
        return state["handle"].run()
    x.grad = y.grad = None
    D = dtw_matrix(x, y, case["r"])
    soft_assignment_loss(D).backward()
    return {"distances": D.detach(), "grad_x": x.grad, "grad_y": y.grad}


# --------------------------------------------------------------------------
# work


def _half_width(n, m, r):
    return int(max(math.floor(min(n, m) * r), 1))


def _band_cells(n, m, r):
    w = _half_width(n, m, r)
    mx, mn = max(0, m - n) + w, max(0, n - m)
    i = np.arange(n)
    return int((np.minimum(m, i + mx) - np.maximum(0, i - mn - w + 1)).sum())


# arithmetic of one cell of the recurrence, minima not counted
_CELL = {"dtw": 3, "ddtw": 3, "wdtw": 4, "adtw": 4, "lcss": 2, "edr": 2, "erp": 4, "msm": 8,
         "twe": 9}


def work(case):
    f = case["family"]
    if f in ("pairwise", "edit"):
        lx, ly = case["lx"], case["ly"]
        cells = _band_cells(lx, ly, case.get("r", 1.0))
        return {"bytes": 8.0 * (case["nx"] * lx + case["ny"] * ly + case["nx"] * case["ny"]),
                "flops": float(_CELL[case["metric"]]) * cells * case["nx"] * case["ny"]}
    if f == "euclidean":
        L = case["length"]
        return {"bytes": 8.0 * ((case["nx"] + case["ny"]) * L + case["nx"] * case["ny"]),
                "flops": 3.0 * case["nx"] * case["ny"] * L}
    if f == "argmin":
        L = case["length"]
        return {"bytes": 8.0 * ((case["nx"] + case["ny"]) * L + 2 * case["nx"] * case["k"]),
                "flops": 3.0 * case["nx"] * case["ny"] * _band_cells(L, L, case["r"])}
    if f == "subsequence":
        lens = np.arange(case["low"], case["high"] + 1)
        windows = case["length"] - lens + 1
        if case["metric"] == "dtw":
            per = np.array([3.0 * _band_cells(int(v), int(v), case["r"]) for v in lens])
        else:
            per = 3.0 * lens
        return {"bytes": 8.0 * (case["m"] * float(lens.mean()) + case["n"] * case["length"] +
                                2 * case["n"] * case["m"]),
                "flops": float((per * windows).mean()) * case["m"] * case["n"]}
    if f == "batched":
        # the mean over uniformly spread lengths, sampled on a grid
        grid = np.linspace(case["low"], case["high"], 12).astype(int)
        cells = np.mean([_band_cells(int(a), int(b), case["r"]) for a in grid for b in grid])
        return {"bytes": 4.0 * case["n"] * case["dims"] * (case["low"] + case["high"]) +
                8.0 * case["n"],
                "flops": 3.0 * float(cells) * case["n"] * case["dims"]}
    L = case["length"]
    return {"bytes": 8.0 * (case["nx"] + case["ny"]) * L + 8.0 * case["nx"] * case["ny"],
            "flops": 3.0 * case["nx"] * case["ny"] * _band_cells(L, L, case["r"])}


# --------------------------------------------------------------------------
# results in 64 bits


def _sweep(X, Y, n, m, band, row0, col0, corner, border, cell):
    """Final cell of a banded recurrence for every row pair of X (P, n), Y (P, m).

    Runs anti-diagonal by anti-diagonal over the rows that can be in band.
    ``cell(i, j, diag, up, left)`` gives the new values of rows i (int tensor)
    at columns j = d - i.  Neighbours above row 0 / left of column 0 are
    row0 / col0 (with ``corner`` at (-1, -1)); neighbours out of band read
    ``border``.
    """
    P = X.shape[0]
    dev = X.device
    mx, mn = max(0, m - n) + band, max(0, n - m)
    prev = prev2 = None  # (first row, values (P, rows))

    def at(state, rows, fill):
        out = torch.full((P, rows.numel()), fill, dtype=torch.float64, device=dev)
        if state is not None:
            lo, v = state
            a = max(int(rows[0]), lo)
            b = min(int(rows[-1]), lo + v.shape[1] - 1)
            if a <= b:
                out[:, a - int(rows[0]):b + 1 - int(rows[0])] = v[:, a - lo:b + 1 - lo]
        return out

    result = None
    for d in range(n + m - 1):
        # rows i with j = d - i in [max(0, i - mn - band + 1), min(m, i + mx))
        lo = max(0, d - m + 1, (d - mx) // 2 + 1)
        hi = min(n - 1, d, (d + mn + band - 1) // 2)
        if lo > hi:
            prev2, prev = prev, None
            continue
        rows = torch.arange(lo, hi + 1)
        i = rows.to(dev)
        j = d - i
        up = at(prev, rows - 1, border)
        left = at(prev, rows, border)
        diag = at(prev2, rows - 1, border)
        if lo == 0:
            up[:, 0] = row0[:, d] if torch.is_tensor(row0) else row0
            diag[:, 0] = (row0[:, d - 1] if torch.is_tensor(row0) else row0) if d else corner
        if hi == d:
            left[:, -1] = col0[:, d] if torch.is_tensor(col0) else col0
            if d > 0:
                diag[:, -1] = col0[:, d - 1] if torch.is_tensor(col0) else col0
        value = cell(i, j, diag, up, left)
        if d == n + m - 2:
            result = value[:, -1]
        prev2, prev = prev, (lo, value)
    return result


def _slopes(A):
    return ((A[..., 1:-1] - A[..., :-2]) + (A[..., 2:] - A[..., :-2]) / 2) / 2


def _elastic(metric, X, Y, params, r):
    """Distances of the row pairs of X (P, n) and Y (P, m), float64 CUDA."""
    inf = math.inf
    band = _half_width(X.shape[1], Y.shape[1], r)
    if metric == "ddtw":
        X, Y = _slopes(X), _slopes(Y)
    n, m = X.shape[1], Y.shape[1]
    dev = X.device
    if metric in ("dtw", "ddtw"):
        def cell(i, j, diag, up, left):
            return torch.minimum(torch.minimum(up, left), diag) + (X[:, i] - Y[:, j]) ** 2
        return torch.sqrt(_sweep(X, Y, n, m, band, inf, inf, 0.0, inf, cell))
    if metric == "wdtw":
        k = np.arange(max(n, m), dtype=np.float64)
        w = torch.as_tensor(1.0 / (1.0 + np.exp(-0.05 * (k - max(n, m) / 2.0))), device=dev)

        def cell(i, j, diag, up, left):
            # the first row weighs column j with index j - 1
            at = torch.where(i == 0, (j - 1).clamp(min=0), (i - j).abs())
            return (torch.minimum(torch.minimum(up, left), diag) +
                    (X[:, i] - Y[:, j]) ** 2 * w[at])
        return torch.sqrt(_sweep(X, Y, n, m, band, inf, inf, 0.0, inf, cell))
    if metric == "adtw":
        def cell(i, j, diag, up, left):
            move = torch.minimum(up, left) + 1.0
            move = torch.where(i == 0, left, move)  # the first row moves without a penalty
            return torch.minimum(move, diag) + (X[:, i] - Y[:, j]) ** 2
        return torch.sqrt(_sweep(X, Y, n, m, band, inf, inf, 0.0, inf, cell))
    if metric == "lcss":
        def cell(i, j, diag, up, left):
            match = (X[:, i] - Y[:, j]).abs() <= params["epsilon"]
            return torch.where(match, diag + 1.0, torch.maximum(left, up))
        v = _sweep(X, Y, n, m, band, 0.0, 0.0, 0.0, 0.0, cell)
        return 1.0 - v / min(n, m)
    if metric == "edr":
        def cell(i, j, diag, up, left):
            match = (X[:, i] - Y[:, j]).abs() < params["epsilon"]
            return torch.minimum(torch.where(match, diag, diag + 1.0),
                                 torch.minimum(up, left) + 1.0)
        return _sweep(X, Y, n, m, band, 0.0, 0.0, 0.0, 0.0, cell) / max(n, m)
    if metric == "erp":
        gx, gy = X.abs(), Y.abs()  # gap value 0
        sx = torch.zeros(X.shape[0], 1, dtype=torch.float64, device=dev)
        sy = torch.zeros_like(sx)
        for k in range(n):
            sx = sx + gx[:, k:k + 1]
        for k in range(m):
            sy = sy + gy[:, k:k + 1]

        def cell(i, j, diag, up, left):
            return torch.minimum(torch.minimum(diag + (X[:, i] - Y[:, j]).abs(), up + gx[:, i]),
                                 left + gy[:, j])
        return _sweep(X, Y, n, m, band, sy.expand(-1, m), sx.expand(-1, n), 0.0, 0.0, cell)
    if metric == "twe":
        Xp = torch.cat([torch.zeros_like(X[:, :1]), X[:, :-1]], 1)
        Yp = torch.cat([torch.zeros_like(Y[:, :1]), Y[:, :-1]], 1)
        nu, lam = 0.001, 1.0

        def cell(i, j, diag, up, left):
            gap = torch.minimum(up + (Xp[:, i] - X[:, i]).abs(),
                                left + (Yp[:, j] - Y[:, j]).abs()) + (lam + nu)
            match = (diag + (X[:, i] - Y[:, j]).abs() + (Xp[:, i] - Yp[:, j]).abs() +
                     2 * nu * (i - j).abs())
            return torch.minimum(gap, match)
        return _sweep(X, Y, n, m, band, inf, inf, 0.0, 0.0, cell)
    # msm: the split / merge costs are formed in float32, as the reference does
    Xf, Yf = X.float(), Y.float()

    def move(x, y, z):
        inside = ((y <= x) & (x <= z)) | ((y >= x) & (x >= z))
        extra = torch.minimum((x - y).abs(), (x - z).abs())
        return 1.0 + torch.where(inside, torch.zeros_like(extra), extra).double()

    def cell(i, j, diag, up, left):
        xi, yj = Xf[:, i], Yf[:, j]
        xq, yq = Xf[:, (i - 1).clamp(min=0)], Yf[:, (j - 1).clamp(min=0)]
        return torch.minimum(torch.minimum(diag + (X[:, i] - Y[:, j]).abs(),
                                           up + move(xi, xq, yj)), left + move(yj, xi, yq))
    return _sweep(X, Y, n, m, band, inf, inf, 0.0, inf, cell)


def _all_pairs(metric, X, Y, params, r):
    X = torch.as_tensor(X, dtype=torch.float64, device="cuda")
    Y = torch.as_tensor(Y, dtype=torch.float64, device="cuda")
    out = torch.empty(X.shape[0], Y.shape[0], dtype=torch.float64, device="cuda")
    step = max(1, (1 << 19) // Y.shape[0])
    for a in range(0, X.shape[0], step):
        x = X[a:a + step]
        px = x.repeat_interleave(Y.shape[0], 0)
        py = Y.repeat(x.shape[0], 1)
        out[a:a + step] = _elastic(metric, px, py, params, r).view(x.shape[0], -1)
    return out


def _exact_subsequence(case, shapelets, x):
    X = torch.as_tensor(x, device="cuda")
    scaled = case["metric"] == "scaled_euclidean"
    dist = torch.empty(X.shape[0], len(shapelets), dtype=torch.float64, device="cuda")
    index = torch.empty(X.shape[0], len(shapelets), dtype=torch.int64, device="cuda")
    lens = np.array([len(s) for s in shapelets])
    for L in np.unique(lens):
        at = np.flatnonzero(lens == L)
        S = torch.as_tensor(np.stack([shapelets[i] for i in at]), device="cuda")
        W = X.unfold(1, int(L), 1)  # (n, windows, L)
        if scaled:
            S = (S - S.mean(1, keepdim=True)) / S.std(1, correction=0, keepdim=True)
            W = (W - W.mean(2, keepdim=True)) / W.std(2, correction=0, keepdim=True)
        for s, i in zip(S, at):
            if case["metric"] == "dtw":
                flat = W.reshape(-1, int(L))
                d = _elastic("dtw", s[None].expand(flat.shape[0], -1), flat, {}, case["r"])
                d = d.view(W.shape[0], W.shape[1])
            else:
                d = ((W - s) ** 2).sum(2).sqrt()
            dist[:, i], index[:, i] = d.min(1)
    return {"distances": dist, "indices": index}


def _exact_batched(case, x, y):
    n, dims, width = x.shape
    X = torch.as_tensor(x.reshape(n * dims, width), device="cuda").double()
    Y = torch.as_tensor(y.reshape(n * dims, width), device="cuda").double()
    nl = (~X.isnan()).sum(1)
    ml = (~Y.isnan()).sum(1)
    X, Y = X.nan_to_num(0.0), Y.nan_to_num(0.0)
    out = torch.empty(n * dims, dtype=torch.float64, device="cuda")
    order = torch.argsort(torch.maximum(nl, ml))
    for part in order.split(2048):
        a, b = nl[part, None], ml[part, None]
        band = torch.clamp(torch.floor(torch.minimum(a, b) * case["r"]), min=1).long()
        mx, mn = (b - a).clamp(min=0) + band, (a - b).clamp(min=0)
        N, M = int(a.max()), int(b.max())
        px, py = X[part], Y[part]
        i = torch.arange(N, device="cuda")[None, :]
        inf = torch.full((part.numel(), N + 1), math.inf, dtype=torch.float64, device="cuda")
        prev, prev2 = inf.clone(), inf.clone()  # value of row i at position i + 1
        found = torch.empty(part.numel(), dtype=torch.float64, device="cuda")
        for d in range(N + M - 1):
            j = d - i
            ok = ((i < a) & (j >= 0) & (j < b) & (j >= i - mn - band + 1) & (j < i + mx))
            best = torch.minimum(torch.minimum(prev[:, :-1], prev[:, 1:]), prev2[:, :-1])
            if d == 0:
                best[:, 0] = 0.0
            lo, hi = max(0, d - N + 1), min(M - 1, d)
            row = torch.zeros_like(px[:, :N])
            row[:, d - hi:d - lo + 1] = py[:, lo:hi + 1].flip(1)
            value = torch.where(ok, best + (px[:, :N] - row) ** 2, inf[:, 1:])
            last = (a + b - 2 == d).squeeze(1)
            if bool(last.any()):
                found[last] = value[last].gather(1, a[last] - 1).squeeze(1)
            prev2, prev = prev, torch.cat([inf[:, :1], value], 1)
        out[part] = found.sqrt()
    return out.view(n, dims).mean(1)


def _exact_gradient(case, x, c):
    """Distances and gradients along each pair's best path (diagonal moves
    first among equals)."""
    X = torch.as_tensor(x, device="cuda").double()
    C = torch.as_tensor(c, device="cuda").double()
    L, k = X.shape[1], C.shape[0]
    band = _half_width(L, L, case["r"])
    D = _all_pairs("dtw", X, C, {}, case["r"]).requires_grad_(True)
    (G,) = torch.autograd.grad(soft_assignment_loss(D), D)
    D = D.detach()
    gx, gc = torch.zeros_like(X), torch.zeros_like(C)
    ninf = math.inf
    for a in range(0, X.shape[0], max(1, (1 << 15) // k)):
        xs = X[a:a + max(1, (1 << 15) // k)]
        P = xs.shape[0] * k
        px, pc = xs.repeat_interleave(k, 0), C.repeat(xs.shape[0], 1)
        moves = torch.empty(2 * L - 1, P, L, dtype=torch.uint8, device="cuda")
        i = torch.arange(L, device="cuda")
        prev = torch.full((P, L + 1), ninf, dtype=torch.float64, device="cuda")
        prev2 = prev.clone()
        for d in range(2 * L - 1):
            j = d - i
            ok = (j >= 0) & (j < L) & ((i - j).abs() < band)
            diag, up, left = prev2[:, :-1], prev[:, :-1], prev[:, 1:]
            best, move = diag, torch.zeros(P, L, dtype=torch.uint8, device="cuda")
            move = torch.where(up < best, torch.ones_like(move), move)
            best = torch.minimum(best, up)
            move = torch.where(left < best, torch.full_like(move, 2), move)
            best = torch.minimum(best, left)
            moves[d] = move
            if d == 0:
                best = best.clone()
                best[:, 0] = 0.0
            v = best + (px - pc[:, j.clamp(0, L - 1)]) ** 2
            v = torch.where(ok, v, torch.full_like(v, ninf))
            prev2, prev = prev, torch.cat([torch.full_like(v[:, :1], ninf), v], 1)
        up_g = (G[a:a + xs.shape[0]] / D[a:a + xs.shape[0]]).reshape(-1)
        who = torch.arange(P, device="cuda")
        r = torch.full((P,), L - 1, device="cuda")
        s = torch.full((P,), L - 1, device="cuda")
        live = torch.ones(P, dtype=torch.bool, device="cuda")
        gpx, gpc = torch.zeros_like(px), torch.zeros_like(pc)
        for _ in range(2 * L - 1):
            term = torch.where(live, up_g * (px[who, r] - pc[who, s]), torch.zeros_like(up_g))
            gpx[who, r] += term
            gpc[who, s] -= term
            move = moves[r + s, who, r]
            live &= (r + s) > 0
            r = torch.where(live & (move != 2), r - 1, r)
            s = torch.where(live & (move != 1), s - 1, s)
        gx[a:a + xs.shape[0]] = gpx.view(-1, k, L).sum(1)
        gc += gpc.view(-1, k, L).sum(0)
    return {"distances": D, "grad_x": gx, "grad_y": gc}


def exact(case, seed):
    a, b = _arrays(case, seed)
    f = case["family"]
    if f in ("pairwise", "edit"):
        out = _all_pairs(case["metric"], a, b, _params(case), case.get("r", 1.0))
        out = out.squeeze()
        return out.cpu().numpy() if case.get("host") else out
    if f == "euclidean":
        X, Y = torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda")
        out = torch.zeros(X.shape[0], Y.shape[0], dtype=torch.float64, device="cuda")
        for k in range(X.shape[1]):
            out += (Y[None, :, k] - X[:, None, k]) ** 2
        return out.sqrt().squeeze()
    if f == "argmin":
        D = _all_pairs("dtw", a, b, {}, case["r"])
        distances, indices = torch.sort(D, dim=1, stable=True)
        k = min(case["k"], D.shape[1])
        return {"indices": indices[:, :k].contiguous(),
                "distances": distances[:, :k].contiguous()}
    if f == "subsequence":
        # a sweep per shapelet length and pair of diagonals: bounded by the
        # number of shapelets
        if case["metric"] == "dtw" and case["m"] > 400:
            return None
        return _exact_subsequence(case, a, b)
    if f == "batched":
        return _exact_batched(case, a, b)
    return _exact_gradient(case, a, b)
