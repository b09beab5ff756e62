"""The work that users of this framework have it do, as measurable cases.

Each case is one pass through a public entry point: the kNN graph (exact and
NNDescent), the fuzzy set with the spectral start, the layout epochs, one training
step and the transform of the learned encoder, and a whole small fit.  Sizes are those
of the repository's own workloads (2,000 x 64; 20,000 x 784; 70,000 x 784;
1,000,000 x 128), or generic ones around them.  `listed` gives the fixed cases, `draw`
more of the same ranges, `exact` the same results in 64 bits from plain torch.

A layout that runs for hundreds of epochs at full step size amplifies the last bit of
a sum to a visible move, so that no two runs can be compared.  The layout cases
therefore run the last part of a fit with a small learning rate, and the whole fit is a
short one with a small learning rate; the work per epoch is that of any other epoch.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from mlx_vis_b200 import UMAP, NNDescent, _lib
from mlx_vis_b200._knn import knn_device
from mlx_vis_b200.encoder import Encoder

DEV = "cuda"
# the membership curve of min_dist 0.1, spread 1 (the defaults)
CURVE_A, CURVE_B = 1.5769434603113077, 0.8950608779109733
LAYOUT_SEED = 0x9E3779B97F4A7C15
LAYOUT_RATE = 0.25
HIDDEN = 512


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a small exploratory data set: the exact graph is a few launches
        {"name": "knn_2k", "kind": "knn", "n": 2000, "d": 64, "k": 15, "data": "clusters"},
        # features already reduced to 50, a wider neighbourhood, odd row count
        {"name": "knn_10k_k30", "kind": "knn", "n": 9999, "d": 50, "k": 30, "data": "clusters"},
        # images at the largest size the automatic choice computes exactly
        {"name": "knn_20k", "kind": "knn", "n": 20000, "d": 784, "k": 15, "data": "pixels"},
        # the approximate graph: a wider neighbourhood on reduced features, whose length is
        # not a multiple of four
        {"name": "nnd_30k_k30", "kind": "nnd", "n": 30001, "d": 50, "k": 30, "data": "clusters"},
        # ... the 70,000 image workload
        {"name": "nnd_70k", "kind": "nnd", "n": 70000, "d": 784, "k": 15, "data": "pixels"},
        # ... the largest workload, a million rows
        {"name": "nnd_1m", "kind": "nnd", "n": 1000000, "d": 128, "k": 15, "data": "clusters"},
        # the graph's weights and the spectral start at the image workload's size
        {"name": "graph_70k", "kind": "graph", "n": 70000, "k": 15, "dim": 2, "epochs": 500},
        # layout epochs of a small fit, where launches count
        {"name": "layout_2k", "kind": "layout", "n": 2000, "k": 15, "dim": 2, "epochs": 500, "begin": 450, "neg": 5},
        # layout epochs at the image workload's size
        {"name": "layout_70k", "kind": "layout", "n": 70000, "k": 15, "dim": 2, "epochs": 500, "begin": 450, "neg": 5},
        # the learned start: one training step at its default batch
        {"name": "train_4k", "kind": "train", "n": 4096, "d": 784, "dim": 2},
        # ... and the embedding of the whole image workload by the trained encoder
        {"name": "transform_70k", "kind": "transform", "n": 70000, "d": 784, "dim": 2},
        # a whole small fit from a host array to a host embedding
        {"name": "fit_2k", "kind": "fit", "n": 2000, "d": 64, "k": 15, "dim": 2, "epochs": 25, "data": "clusters"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["knn", "knn", "nnd", "nnd", "graph", "layout", "layout", "train", "transform", "fit"])
    data = rng.choice(["clusters", "pixels"])
    if kind == "knn":
        return {"kind": kind, "n": _log_int(rng, 300, 20000), "d": _log_int(rng, 8, 1024),
                "k": rng.choice([5, 10, 15, 15, 20, 30, 50, 100]), "data": data}
    if kind == "nnd":
        while True:  # no more work than the million rows
            c = {"kind": kind, "n": _log_int(rng, 20001, 300000), "d": _log_int(rng, 16, 1024),
                 "k": rng.choice([5, 10, 15, 15, 20, 30, 50]), "data": data}
            if c["n"] * c["k"] ** 2 * (1 + c["d"] / 400) <= 8e7:
                return c
    if kind == "graph":
        return {"kind": kind, "n": _log_int(rng, 500, 300000), "k": rng.choice([5, 10, 15, 15, 20, 30, 50]),
                "dim": rng.choice([2, 2, 3]), "epochs": rng.choice([200, 500])}
    if kind == "layout":
        epochs = rng.choice([200, 500])
        return {"kind": kind, "n": _log_int(rng, 500, 300000), "k": rng.choice([5, 10, 15, 15, 20, 30]),
                "dim": rng.choice([2, 2, 3]), "epochs": epochs, "begin": int(epochs * rng.uniform(0.88, 0.94)),
                "neg": rng.choice([5, 5, 5, 3, 10])}
    if kind == "train":
        return {"kind": kind, "n": _log_int(rng, 200, 8192), "d": _log_int(rng, 16, 1024), "dim": rng.choice([2, 2, 3])}
    if kind == "transform":
        return {"kind": kind, "n": _log_int(rng, 1, 200000), "d": _log_int(rng, 16, 1024), "dim": rng.choice([2, 2, 3])}
    return {"kind": kind, "n": _log_int(rng, 300, 6000), "d": _log_int(rng, 8, 256), "k": rng.choice([5, 10, 15, 15, 30]),
            "dim": rng.choice([2, 2, 3]), "epochs": 25, "data": data}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rows(n, d, data, g):
    """Feature rows: pixel-like mixtures of 10 prototypes (about half the entries zero, noise
    0.1, clipped to [0, 1]) or 100 anisotropic Gaussian clusters."""
    if data == "pixels":
        protos = torch.rand(10, d, device=DEV, generator=g)
        protos = protos * (torch.rand(10, d, device=DEV, generator=g) >= 0.5)
        label = torch.randint(0, 10, (n,), device=DEV, generator=g)
        return (protos[label] + 0.1 * torch.randn(n, d, device=DEV, generator=g)).clamp_(0, 1)
    centres = 4.0 * torch.randn(100, d, device=DEV, generator=g)
    scale = 0.3 + 1.7 * torch.rand(100, d, device=DEV, generator=g)
    label = torch.randint(0, 100, (n,), device=DEV, generator=g)
    return centres[label] + scale[label] * torch.randn(n, d, device=DEV, generator=g)


def _knn_graph(n, k, g):
    """A kNN graph with the structure of a real one, without a kNN search over all rows:
    rows in groups of about 500, exact neighbours inside the group in a 6-d latent space,
    2% of the rows with a last neighbour in some other group, and the rows in random order.
    Returns (idx int32, dist float32 ascending, latent rows, group of each row)."""
    groups = max(1, n // 500)
    size = -(-n // groups)
    row = torch.arange(groups, device=DEV)[:, None] + groups * torch.arange(size, device=DEV)[None, :]
    inside = row < n
    z = torch.randn(groups, size, 6, device=DEV, generator=g)
    idx = torch.empty(n, k, dtype=torch.int64, device=DEV)
    dist = torch.empty(n, k, device=DEV)
    for b in range(0, groups, 64):  # 64 groups at a time
        zb, ib, rb = z[b:b + 64], inside[b:b + 64], row[b:b + 64]
        d2 = (zb[:, :, None, :] - zb[:, None, :, :]).square().sum(-1)
        d2 = d2.masked_fill(~ib[:, None, :], float("inf"))
        d2.diagonal(dim1=1, dim2=2).fill_(float("inf"))
        val, pos = d2.topk(k, dim=2, largest=False)
        nb = torch.gather(rb[:, None, :].expand(-1, size, -1), 2, pos)
        idx[rb[ib]] = nb[ib]
        dist[rb[ib]] = (val[ib] + 4.0).sqrt()
    if groups > 1:  # a link to another group
        far = torch.rand(n, device=DEV, generator=g) < 0.02
        own = torch.arange(n, device=DEV) % groups
        step = torch.randint(1, groups, (n,), device=DEV, generator=g)
        other = (own + step) % groups  # row `other` is the first row of that group
        idx[:, -1] = torch.where(far, other, idx[:, -1])
    order = torch.randperm(n, device=DEV, generator=g)  # new id of each row
    out_i, out_d = torch.empty_like(idx), torch.empty_like(dist)
    out_i[order] = order[idx]
    out_d[order] = dist
    latent = torch.empty(n, 6, device=DEV)
    latent[order[row[inside]]] = z[inside]
    group = torch.empty(n, dtype=torch.int64, device=DEV)
    group[order] = torch.arange(n, device=DEV) % groups
    return out_i.int().contiguous(), out_d.contiguous(), latent, group


def _fuzzy64(idx, dist, epochs):
    """The fuzzy set in 64 bits: (rows, cols, weights), the rows' edges in list order."""
    n, k = idx.shape
    d = dist.double()
    rho = torch.where(d > 0, d, torch.full_like(d, float("inf"))).amin(1, keepdim=True).clamp_min(1e-8)
    gap = (d - rho).clamp_min(0)
    target = math.log2(k)
    lo = torch.full((n, 1), 1e-20, dtype=torch.float64, device=DEV)
    hi = torch.full_like(lo, 1e3)
    sigma = torch.ones_like(lo)
    done = torch.zeros_like(lo, dtype=torch.bool)
    for _ in range(64):
        s = torch.exp(-gap[:, 1:] / sigma).sum(1, keepdim=True)
        done = done | ((s - target).abs() < 1e-5)
        up, down = (s > target) & ~done, (s < target) & ~done
        hi = torch.where(up, sigma, hi)
        lo = torch.where(down, sigma, lo)
        grown = torch.where(hi >= 1e3, sigma * 2, (sigma + hi) / 2)
        sigma = torch.where(up, (lo + sigma) / 2, torch.where(down, grown, sigma))
    w = torch.exp(-gap / sigma.clamp_min(1e-10)).float().double()
    own = torch.arange(n, device=DEV)
    sym = torch.empty_like(w)
    for b in range(0, n, 20000):  # the weight of the opposite edge, where there is one
        j = idx[b:b + 20000].long()
        hit = idx[j].long() == own[b:b + 20000, None, None]
        first = hit.int().argmax(2)
        back = torch.where(hit.any(2), torch.gather(w[j], 2, first[:, :, None])[:, :, 0], torch.zeros_like(w[b:b + 20000]))
        wb = w[b:b + 20000]
        sym[b:b + 20000] = wb + back - wb * back
    sym = sym.float()
    keep = sym >= sym.max() / epochs
    return own[:, None].expand(n, k)[keep], idx.long()[keep], sym[keep]


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind in ("knn", "nnd"):
        X = _rows(case["n"], case["d"], case["data"], g).contiguous()
        return {"kind": kind, "X": X, "k": case["k"], "seed": int(seed) % 100000}
    if kind == "graph":
        n, dim = case["n"], case["dim"]
        idx, dist, _, _ = _knn_graph(n, case["k"], g)
        return {"kind": kind, "idx": idx, "dist": dist, "n": n, "dim": dim, "epochs": case["epochs"],
                "V0": torch.randn(n, dim + 1, device=DEV, generator=g),
                "noise": 1e-4 * torch.randn(n, dim, device=DEV, generator=g)}
    if kind == "layout":
        n, k, dim = case["n"], case["k"], case["dim"]
        idx, dist, latent, group = _knn_graph(n, k, g)
        r, c, w = _fuzzy64(idx, dist, case["epochs"])
        rows = torch.zeros(n * k, dtype=torch.int32, device=DEV)  # room for every directed edge, as after a fit's kNN
        cols, vals = torch.zeros_like(rows), torch.zeros(n * k, device=DEV)
        rows[:r.numel()], cols[:r.numel()], vals[:r.numel()] = r.int(), c.int(), w
        centre = 30.0 * torch.rand(int(group.max()) + 1, dim, device=DEV, generator=g)
        Y0 = (centre[group] + 0.5 * latent[:, :dim]).contiguous()
        n_edges = torch.full((1,), r.numel(), dtype=torch.int64, device=DEV)
        # the schedule as it stands when the epochs before `begin` are done
        eps = torch.div(torch.tensor(float(case["epochs"]), device=DEV), case["epochs"] * (w / w.max()))
        due = eps.clone()
        for e in range(case["begin"]):
            due = torch.where(due <= e, due + eps, due)
        due_all = torch.zeros(n * k, device=DEV)
        due_all[:due.numel()] = due
        lay = _lib.Layout(rows, cols, vals, n_edges, n, dim, case["epochs"])
        return {"kind": kind, "lay": lay, "Y0": Y0, "Y": Y0.clone(), "due": due_all, "begin": case["begin"],
                "end": case["epochs"], "neg": case["neg"], "eps": eps, "rows": r, "cols": c}
    if kind in ("train", "transform"):
        enc = Encoder(case["d"], hidden=HIDDEN, out_dim=case["dim"], seed=int(seed) % 100000)
        X = _rows(case["n"], case["d"], "pixels", g).contiguous()
        if kind == "train":
            T = torch.randn(case["n"], case["dim"], device=DEV, generator=g)
            return {"kind": kind, "enc": enc, "X": X, "T": T}
        enc.y_scale_ = (torch.randn(case["dim"], device=DEV, generator=g),
                        5.0 + torch.rand(case["dim"], device=DEV, generator=g))
        return {"kind": kind, "enc": enc, "X": X}
    X = _rows(case["n"], case["d"], case["data"], g).cpu().numpy()
    return {"kind": kind, "X": X, "k": case["k"], "dim": case["dim"], "epochs": case["epochs"],
            "seed": int(seed) % 100000}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "knn":
        return knn_device(state["X"], state["k"], method="brute")
    if kind == "nnd":
        return NNDescent(k=state["k"], random_state=state["seed"]).build_device(state["X"])
    if kind == "graph":
        rows, cols, vals, n_edges = _lib.fuzzy(state["idx"], state["dist"], state["epochs"])
        Y = _lib.spectral(rows, cols, vals, n_edges, state["n"], state["dim"], state["V0"], state["noise"],
                          n_iter=100, fallback_seed=1)
        return Y, n_edges
    if kind == "layout":
        lay, Y = state["lay"], state["Y"]
        lay.next.copy_(state["due"])
        Y.copy_(state["Y0"])
        lay.epochs(Y, state["begin"], state["end"], CURVE_A, CURVE_B, LAYOUT_RATE, state["neg"], LAYOUT_SEED, graph=True)
        return Y
    if kind == "train":
        enc = state["enc"]
        loss = enc.train_step(state["X"], state["T"])
        return {"loss": loss, "grads": dict(enc.grads), "params": dict(enc.params)}
    if kind == "transform":
        return state["enc"].transform_device(state["X"])
    return UMAP(n_components=state["dim"], n_neighbors=state["k"], n_epochs=state["epochs"], learning_rate=0.05,
                knn_method="brute", random_state=state["seed"]).fit_transform(state["X"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind, n = case["kind"], case["n"]
    k, d, dim = case.get("k", 0), case.get("d", 0), case.get("dim", 2)
    if kind == "knn":
        return {"bytes": 4 * n * d + 8 * n * k, "flops": 2 * n * n * d}
    if kind == "nnd":  # one join of every row with its neighbours' neighbours
        return {"bytes": 4 * n * d + 8 * n * k, "flops": 2 * n * k * k * d}
    if kind == "graph":  # the graph in, the edges once, V once in each direction for each of 100 steps
        return {"bytes": 20 * n * k + 100 * (8 * n * k + 8 * n * (dim + 1)) + 4 * n * dim,
                "flops": 100 * n * (dim + 1) * (2 * k + 2 * (dim + 1))}
    if kind == "layout":  # about 0.36 of the edges are due in an epoch: ids, schedule, positions, moves
        due = 0.36 * n * k * (case["epochs"] - case["begin"])
        return {"bytes": due * (16 + 4 * dim * (2 + case["neg"]) + 16 * dim), "flops": due * 20 * (1 + case["neg"])}
    if kind == "train":
        weights = HIDDEN * (d + HIDDEN + dim)
        return {"bytes": 4 * n * (d + dim) + 28 * weights, "flops": 6 * n * weights}
    if kind == "transform":
        weights = HIDDEN * (d + HIDDEN + dim)
        return {"bytes": 4 * n * (d + dim) + 2 * weights, "flops": 2 * n * weights}
    return {"bytes": 4 * n * d + 100 * 8 * n * k + case["epochs"] * 0.36 * n * k * 112, "flops": 2 * n * n * d}


def tolerance(case):
    kind = case["kind"]
    if kind == "knn":  # FP32 distances; a tie within their rounding may come in either order
        return {"rel": 2e-6, "max": 2e-5, "differ": 1e-3}
    if kind == "nnd":  # with its sums in another order the search keeps all but 0.35% of the entries (rel 1e-4, max 0.02)
        return {"rel": 4e-4, "max": 0.08, "differ": 0.01}
    if kind == "graph":  # against 64 bits: rel 5e-7, max 2e-6
        return {"rel": 2e-6, "max": 1e-5}
    if kind == "layout":  # sums in another order: rel 2e-5, max 4e-4 at most, mostly below 1e-7 and 1e-5
        return {"rel": 6e-5, "max": 1.5e-3}
    if kind == "train":  # BF16 operands: 3e-3 against 64 bits; AdamW's first step moves by the gradient's sign
        return {"rel": 1e-2, "max": 0.2}
    if kind == "transform":  # BF16 operands: rel 3e-3, max 0.01 against 64 bits
        return {"rel": 1e-2, "max": 0.04}
    return {"rel": 1e-3, "max": 2e-2}  # sums in another order: rel 2.3e-4, max 5e-3 at most


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _philox(c0, c1, c2, c3, key):
    """Philox4x32-10 on int64 tensors that hold 32-bit words."""
    mask = 0xFFFFFFFF
    k0, k1 = key & mask, (key >> 32) & mask

    def mulhilo(m, x):  # 32 x 32 -> 64 in two halves, so that nothing leaves the signed range
        lo16, hi16 = (x & 0xFFFF) * m, (x >> 16) * m
        s = (hi16 << 16) & 0xFFFFFFFFFFFF
        total_lo = (lo16 + s) & mask
        hi = (hi16 >> 32 << 16) + ((lo16 + s) >> 32)
        return hi & mask, total_lo

    for _ in range(10):
        hi0, lo0 = mulhilo(0xD2511F53, c0)
        hi1, lo1 = mulhilo(0xCD9E8D57, c2)
        c0, c1, c2, c3 = hi1 ^ c1 ^ k0, lo1, hi0 ^ c3 ^ k1, lo0
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c0, c1, c2, c3


def _layout64(case, s):
    """The epochs in 64 bits, with the schedule's 32-bit recurrence (it decides which edges are due)."""
    n, dim, neg = case["n"], case["dim"], case["neg"]
    a, b = float(np.float32(CURVE_A)), float(np.float32(CURVE_B))
    Y, rows, cols, eps = s["Y0"].double(), s["rows"], s["cols"], s["eps"]
    due_at = s["due"][:eps.numel()].clone()
    edge = torch.arange(eps.numel(), device=DEV)
    for e in range(case["begin"], case["epochs"]):
        act = due_at <= e
        due_at = torch.where(act, due_at + eps, due_at)
        ed = edge[act]
        i, j = rows[act], cols[act]
        alpha = float(np.float32(LAYOUT_RATE * (1.0 - e / case["epochs"])))
        diff = Y[i] - Y[j]
        d2 = diff.square().sum(1, keepdim=True).clamp_min(1e-6)
        coef = -2 * a * b * d2.pow(b) / (d2 * (1 + a * d2.pow(b)))
        move = (coef * diff).clamp(-4, 4) * alpha
        delta = torch.zeros_like(Y)
        delta.index_add_(0, j, -move)
        zero = torch.zeros_like(ed)
        for m in range(neg):
            if m % 4 == 0:
                words = _philox(ed, zero, zero + e, zero + m // 4, LAYOUT_SEED)
            t = (words[m % 4] * n) >> 32
            diff = Y[i] - Y[t]
            d2 = diff.square().sum(1, keepdim=True).clamp_min(1e-6)
            coef = 2 * b / ((0.001 + d2) * (1 + a * d2.pow(b)))
            move = move + (coef * diff).clamp(-4, 4) * alpha
        delta.index_add_(0, i, move)
        Y = Y + delta
    return Y


def _spectral64(case, s):
    n, dim = case["n"], case["dim"]
    rows, cols, w = _fuzzy64(s["idx"], s["dist"], case["epochs"])
    w = w.double()
    deg = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, rows, w).clamp_min(1e-10)
    wn = w * deg[rows].rsqrt() * deg[cols].rsqrt()
    V = s["V0"].double()
    for _ in range(100):
        V = torch.zeros_like(V).index_add_(0, rows, wn[:, None] * V[cols])
        q = []
        for c in range(dim + 1):
            v = V[:, c]
            for u in q:
                v = v - (u @ v) * u
            q.append(v / (v @ v + 1e-10).sqrt())
        V = torch.stack(q, 1)
    e = V[:, 1:]
    e = e * (10.0 / e.abs().max()) + s["noise"].double()
    lo, hi = e.amin(0), e.amax(0)
    return 10.0 * (e - lo) / (hi - lo + 1e-10), torch.tensor([rows.numel()], dtype=torch.int64, device=DEV)


def _forward64(enc, X):
    p = {k: v.double() for k, v in enc.params.items()}
    for v in p.values():
        v.requires_grad_(True)
    h = torch.nn.functional.gelu(X.double() @ p["W1"].T + p["b1"])
    h = torch.nn.functional.gelu(h @ p["W2"].T + p["b2"])
    return h @ p["W3"].T + p["b3"], p


def exact(case, seed):
    kind = case["kind"]
    if kind in ("nnd", "fit"):  # an approximate search, and a layout that follows from every bit before it
        return None
    s = prepare(case, seed)
    if kind == "knn":
        X = s["X"].double()
        sq = X.square().sum(1)
        idx, dist = [], []
        for b in range(0, case["n"], 2000):
            d2 = (sq[b:b + 2000, None] + sq[None, :] - 2.0 * X[b:b + 2000] @ X.T).clamp_min(0)
            own = torch.arange(d2.shape[0], device=DEV)
            d2[own, own + b] = float("inf")
            val, pos = d2.topk(case["k"], dim=1, largest=False)
            idx.append(pos.int())
            dist.append(val.sqrt())
        return torch.cat(idx), torch.cat(dist)
    if kind == "graph":
        return _spectral64(case, s)
    if kind == "layout":
        return _layout64(case, s)
    with torch.enable_grad():
        Y, p = _forward64(s["enc"], s["X"])
        if kind == "transform":
            mean, std = s["enc"].y_scale_
            return (Y * std.double() + mean.double()).detach()
        loss = (Y - s["T"].double()).square().sum(1).mean()
        loss.backward()
    enc = s["enc"]
    new = {}
    for k, v in p.items():  # the first AdamW step: both bias corrections cancel the decay of the averages
        new[k] = (v * (1.0 - enc.lr * enc.wd) - enc.lr * v.grad / (v.grad.abs() + enc.eps)).detach()
    return {"loss": loss.detach().reshape(1), "grads": {k: v.grad for k, v in p.items()}, "params": new}
