"""The work that users of knn_sweet_b200 have it do, as measurable cases.

A case is a dict of plain values.  ``prepare`` makes what a user's program holds
before the call (points on the GPU, offsets, an index, a captured graph),
``run`` is one pass through the public entry points, ``work`` the bytes and
operations no implementation can do without, ``exact`` the same outputs in 64
bits from plain torch.  The kinds:

  join     ``knnjoin`` of device tensors (or of pinned host arrays, ``host``):
           a self-join (m = 0) or a cross join, FP32 or BF16+refine form
  index    ``KnnIndex.query``: a batch of queries against a kept index
  clouds   many point clouds in one call: ``knnjoin_batched``, or
           ``BatchedJoinGraph`` for fixed cloud sizes (``graph``)
  chamfer  one training step: ``knn_chamfer`` (one pair of clouds) or
           ``knn_chamfer_batched``, loss and both gradients

Sizes come from the benchmark configurations (``knn_sweet_b200.data``,
``knn_sweet_b200.workloads``) and the ranges around them.
"""
import math

import numpy as np
import torch

import knn_sweet_b200 as ks
from knn_sweet_b200.autograd import knn_chamfer, knn_chamfer_batched
from knn_sweet_b200.batched import BatchedJoinGraph, knnjoin_batched
from knn_sweet_b200.index import KnnIndex

# exact() is given up beyond this many query-reference pairs (about 20 seconds)
EXACT_PAIRS = 2e11


def _join(name, n, m, d, k, data, *, qreps=0, sreps=0, lloyd=0, trials=10, form="fp32",
          host=False, centers=0):
    return {"name": name, "kind": "join", "n": n, "m": m, "d": d, "k": k, "data": data,
            "qreps": qreps, "sreps": sreps, "lloyd": lloyd, "trials": trials, "form": form,
            "host": host, "centers": centers}


def _clouds(name, clouds, lo, hi, k, *, graph, trials):
    return {"name": name, "kind": "clouds", "clouds": clouds, "lo": lo, "hi": hi, "k": k,
            "graph": graph, "trials": trials}


def _chamfer(name, pairs, lo, hi, k):
    return {"name": name, "kind": "chamfer", "pairs": pairs, "lo": lo, "hi": hi, "k": k}


def listed():
    return [
        # one small point cloud: the smallest call, launches and latency count
        _join("cloud-1k-k16", 1000, 0, 3, 16, "blobs"),
        # the reference's sample run at the size of its table: RGB integers, k = 200
        _join("skin-245k-k200", 245_057, 0, 3, 200, "skin", qreps=800, sreps=800),
        # the drop-in boundary of the reference: host arrays in, host arrays out
        _join("host-skin-100k-k32", 100_003, 0, 3, 32, "skin", host=True),
        # a million 32-wide vectors, both precision forms
        _join("vectors-d32-fp32", 1_000_000, 100_000, 32, 32, "uniform", qreps=1000, sreps=1000,
              lloyd=3, centers=1000),
        _join("vectors-d32-bf16", 1_000_000, 100_000, 32, 32, "uniform", qreps=1000, sreps=1000,
              lloyd=3, form="bf16_refine", centers=1000),
        # 128-wide vectors: the smaller set in FP32, the largest join in the BF16 form
        _join("vectors-d128-fp32", 400_000, 40_000, 128, 100, "normal3", qreps=1600, sreps=1600,
              lloyd=4, centers=800),
        _join("vectors-d128-bf16", 2_000_000, 200_000, 128, 100, "normal3", qreps=8192,
              sreps=8192, lloyd=4, trials=1, form="bf16_refine", centers=4096),
        # a service answering ragged query batches from a kept index
        {"name": "index-d17-k10", "kind": "index", "n": 200_003, "m": 1013, "d": 17, "k": 10,
         "centers": 500},
        # thousands of surface clouds of fixed sizes, one captured graph
        _clouds("clouds-4096-k16", 4096, 256, 16_384, 16, graph=True, trials=1),
        # a small batch of small clouds, sizes new to the caller: a plain call
        _clouds("clouds-64-k16", 64, 256, 2048, 16, graph=False, trials=10),
        # training steps of a nearest-neighbour loss: a batch of pairs, one small pair
        _chamfer("chamfer-64-k8", 64, 2048, 32_768, 8),
        _chamfer("chamfer-1-k1", 1, 1500, 3001, 1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["join3", "join3", "joind", "joind", "index", "clouds", "clouds", "chamfer"])
    if kind == "join3":  # narrow rows: points and colours
        n = _log_int(rng, 500, 245_000)
        c = _join("", n, rng.choice([0, 0, _log_int(rng, 300, n + 300)]), rng.choice([2, 3, 3, 4, 6]),
                  rng.choice([1, 5, 8, 16, 32, 50, 100, 200]), rng.choice(["skin", "blobs"]),
                  host=rng.random() < 0.2)
    elif kind == "joind":  # wide rows: embeddings
        n = _log_int(rng, 5000, 400_000)
        c = _join("", n, max(64, n // rng.randint(4, 12)), rng.choice([16, 24, 31, 48, 64, 100, 128]),
                  rng.choice([1, 10, 32, 50, 100]), rng.choice(["uniform", "normal3"]),
                  lloyd=rng.choice([0, 2, 4]), trials=rng.choice([1, 10]),
                  form=rng.choice(["fp32", "bf16_refine"]), centers=max(8, n // 500))
    elif kind == "index":
        c = {"kind": "index", "n": _log_int(rng, 20_000, 400_000), "m": _log_int(rng, 32, 8000),
             "d": rng.choice([3, 8, 17, 32, 64]), "k": rng.choice([1, 10, 20, 50]), "centers": 500}
    elif kind == "clouds":
        hi = _log_int(rng, 512, 16_384)
        c = _clouds("", _log_int(rng, 8, 1024), max(32, hi // rng.choice([2, 8, 64])), hi,
                    rng.choice([4, 8, 16, 20, 32]), graph=rng.random() < 0.5,
                    trials=rng.choice([1, 10]))
    else:
        hi = _log_int(rng, 1024, 32_768)
        c = _chamfer("", _log_int(rng, 1, 64), hi // 4 + 1, hi, rng.choice([1, 1, 4, 8]))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _mixture(g, centres, sigma, count):
    lab = torch.randint(0, centres.shape[0], (count,), device="cuda", generator=g)
    x = torch.randn((count, centres.shape[1]), device="cuda", generator=g)
    return x.mul_(sigma).add_(centres[lab])


def _skin(g, count, d):
    """Integer colours in [0, 255] from two Gaussians (sigma 40, weights 0.2 / 0.8)."""
    means = torch.tensor([[60.0, 80.0, 140.0], [180.0, 170.0, 160.0]], device="cuda")
    means = means.repeat(1, (d + 2) // 3)[:, :d]
    lab = (torch.rand(count, device="cuda", generator=g) >= 0.2075).long()
    x = torch.randn((count, d), device="cuda", generator=g).mul_(40.0).add_(means[lab])
    return x.round_().clamp_(0.0, 255.0)


def _blobs(g, count, d, blobs=8, sigma=0.05):
    centres = torch.rand((blobs, d), device="cuda", generator=g)
    return _mixture(g, centres, sigma, count).clamp_(0.0, 1.0)


def _points(case, g):
    """(reference points, query points or None for a self-join)."""
    n, m, d = case["n"], case.get("m", 0), case["d"]
    if case["data"] == "skin":
        return _skin(g, n, d), (_skin(g, m, d) if m else None)
    if case["data"] == "blobs":
        both = _blobs(g, n + m, d)  # one draw of centres for both sides
        both = both[torch.randperm(n + m, device="cuda", generator=g)]
        return both[:n].contiguous(), (both[n:].contiguous() if m else None)
    if case["data"] == "uniform":
        centres, sigma = torch.rand((case["centers"], d), device="cuda", generator=g) * 20 - 10, 1.0
    else:
        centres, sigma = torch.randn((case["centers"], d), device="cuda", generator=g) * 3, 0.5
    return _mixture(g, centres, sigma, n), (_mixture(g, centres, sigma, m) if m else None)


def _sizes(case, seed, count):
    """Cloud sizes and their offsets: fixed by the case (the smallest and the
    largest of the range among them), the order by the seed."""
    lo, hi = case["lo"], case["hi"]
    sizes = np.random.default_rng(count * 1_000_003 + hi).integers(lo, hi + 1, size=count)
    sizes[0] = hi
    if count > 1:
        sizes[1] = lo
    np.random.default_rng(seed).shuffle(sizes)
    off = np.zeros(count + 1, np.int64)
    np.cumsum(sizes, out=off[1:])
    return off


def _of_cloud(off):
    counts = torch.as_tensor(np.diff(off)).cuda()
    return torch.repeat_interleave(torch.arange(len(off) - 1, device="cuda"), counts,
                                   output_size=int(off[-1]))


def _surfaces(g, off):
    """Points on randomly shaped ellipsoids, noise 0.01."""
    total, c = int(off[-1]), _of_cloud(off)
    axes = torch.rand((len(off) - 1, 3), device="cuda", generator=g) * 0.8 + 0.2
    v = torch.randn((total, 3), device="cuda", generator=g)
    v /= v.norm(dim=1, keepdim=True)
    return v * axes[c] + 0.01 * torch.randn((total, 3), device="cuda", generator=g)


def _blob_clouds(g, off, blobs=8, sigma=0.05):
    total, c = int(off[-1]), _of_cloud(off)
    centres = torch.rand((len(off) - 1, blobs, 3), device="cuda", generator=g)
    lab = torch.randint(0, blobs, (total,), device="cuda", generator=g)
    x = centres[c, lab] + sigma * torch.randn((total, 3), device="cuda", generator=g)
    return x.clamp_(0.0, 1.0)


def _inputs(case, seed):
    g = _gen(seed)
    if case["kind"] == "join":
        return _points(case, g)
    if case["kind"] == "index":
        return _points(dict(case, data="uniform"), g)
    if case["kind"] == "clouds":
        off = _sizes(case, 0 if case["graph"] else seed, case["clouds"])
        return _surfaces(g, off), off
    xo = _sizes(case, seed, case["pairs"])
    yo = _sizes(case, seed + 1, case["pairs"]) if case["pairs"] > 1 else \
        np.array([0, case["lo"]], np.int64)
    return _blob_clouds(g, xo), xo, _blob_clouds(g, yo), yo


def _pinned(x):
    return x.cpu().pin_memory().numpy()


def prepare(case, seed):
    data = _inputs(case, seed)
    if case["kind"] == "join":
        r, q = data
        if case["host"]:
            m = case["m"] or case["n"]
            out = (torch.empty((m, case["k"]), dtype=torch.int32, pin_memory=True).numpy(),
                   torch.empty((m, case["k"]), dtype=torch.float32, pin_memory=True).numpy())
            return {"case": case, "r": _pinned(r), "q": None if q is None else _pinned(q),
                    "out": out}
        return {"case": case, "r": r, "q": q, "out": None}
    if case["kind"] == "index":
        return {"case": case, "index": KnnIndex(data[0]), "q": data[1]}
    if case["kind"] == "clouds":
        x, off = data
        state = {"case": case, "x": x, "off": off}
        if case["graph"]:
            state["graph"] = BatchedJoinGraph(off, d=3, k=case["k"],
                                              rep_trials=case["trials"]).capture(x)
        return state
    x, xo, y, yo = data
    return {"case": case, "x": x.requires_grad_(True), "xo": xo, "y": y.requires_grad_(True),
            "yo": yo}


def run(state):
    case = state["case"]
    if case["kind"] == "join":
        kw = dict(qreps=case["qreps"], sreps=case["sreps"], rep_trials=case["trials"],
                  lloyd_iters=case["lloyd"], precision=case["form"], out=state["out"])
        if state["q"] is None:
            return ks.knnjoin(state["r"], None, case["k"], **kw)
        return ks.knnjoin(state["q"], state["r"], case["k"], **kw)
    if case["kind"] == "index":
        return state["index"].query(state["q"], case["k"])
    if case["kind"] == "clouds":
        if case["graph"]:
            return state["graph"](state["x"])
        return knnjoin_batched(state["x"], state["off"], k=case["k"], rep_trials=case["trials"])
    x, y = state["x"], state["y"]
    if case["pairs"] == 1:
        loss = knn_chamfer(x, y, case["k"])
    else:
        loss = knn_chamfer_batched(x, state["xo"], y, state["yo"], case["k"])
    gx, gy = torch.autograd.grad(loss, [x, y])
    return loss, gx, gy


def _counts(case):
    """Rows of the two sides (a self-join's points count once) and the queries."""
    if case["kind"] in ("join", "index"):
        return case["n"], case["m"], case["m"] or case["n"]
    if case["kind"] == "clouds":
        n = int(_sizes(case, 0, case["clouds"])[-1])
        return n, 0, n
    n = int(_sizes(case, 0, case["pairs"])[-1])
    m = n if case["pairs"] > 1 else case["lo"]
    return n, m, n + m


def work(case):
    """Inputs read once, results written once, and the distances of the results
    themselves (no join can return them without computing them)."""
    n, m, queries = _counts(case)
    d, k = case.get("d", 3), case["k"]
    out = 4.0 * d * (n + m) + 4.0 if case["kind"] == "chamfer" else 8.0 * k * queries
    flops = 3.0 * d * k * queries
    if case["kind"] == "chamfer":
        flops *= 2.0  # forward and backward
    rows = m if case["kind"] == "index" else n + m
    return {"bytes": 4.0 * d * rows + out, "flops": flops}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
def _nearest(q, r, k):
    """(distances, rows) of the k nearest of r to every row of q, FP64 tensors."""
    m, n, d = q.shape[0], r.shape[0], q.shape[1]
    kk = min(k, n)
    dist = torch.full((m, k), math.inf, dtype=torch.float64, device=q.device)
    rows = torch.full((m, k), -1, dtype=torch.int64, device=q.device)
    step = max(1, int(4e8) // max(n, 1))
    rn = r.square().sum(1)
    for s in range(0, m, step):
        a = q[s:s + step]
        if d <= 8:
            d2 = torch.zeros((a.shape[0], n), dtype=torch.float64, device=q.device)
            for c in range(d):
                d2 += (a[:, c, None] - r[None, :, c]).square_()
            v, i = torch.topk(d2, kk, dim=1, largest=False, sorted=True)
        else:
            # candidates from the expanded form, then their differences
            _, i = torch.topk(torch.addmm(rn[None, :], a, r.T, alpha=-2.0), min(n, kk + 32), dim=1,
                              largest=False, sorted=False)
            v = torch.cat([(a[t:t + 512, None, :] - r[i[t:t + 512]]).square_().sum(2)
                           for t in range(0, a.shape[0], 512)])
            v, o = torch.sort(v, dim=1)
            v, i = v[:, :kk], torch.gather(i, 1, o)[:, :kk]
        dist[s:s + step, :kk] = v.sqrt()
        rows[s:s + step, :kk] = i
    return dist, rows


def _pairs(case):
    if case["kind"] in ("join", "index"):
        return float(case["n"]) * (case["m"] or case["n"])
    off = _sizes(case, 0, case["clouds"] if case["kind"] == "clouds" else case["pairs"])
    return float((np.diff(off).astype(np.float64) ** 2).sum()) * (1 if case["kind"] == "clouds" else 2)


def exact(case, seed):
    if _pairs(case) > EXACT_PAIRS:
        return None
    data = _inputs(case, seed)
    k = case["k"]
    if case["kind"] in ("join", "index"):
        r = data[0].double()
        q = r if data[1] is None else data[1].double()
        return None, _nearest(q, r, k)[0]
    if case["kind"] == "clouds":
        x, off = data[0].double(), data[1]
        return None, torch.cat([_nearest(x[a:b], x[a:b], k)[0] for a, b in zip(off[:-1], off[1:])])
    x, xo, y, yo = data
    x, y = x.double(), y.double()
    gx, gy = torch.zeros_like(x), torch.zeros_like(y)
    loss = torch.zeros((), dtype=torch.float64, device=x.device)
    for p in range(case["pairs"]):
        a, b = slice(int(xo[p]), int(xo[p + 1])), slice(int(yo[p]), int(yo[p + 1]))
        for u, v, gu, gv in ((x[a], y[b], gx[a], gy[b]), (y[b], x[a], gy[b], gx[a])):
            dist, rows = _nearest(u, v, k)
            loss = loss + dist.square().sum()
            diff = 2.0 * (u[:, None, :] - v[rows])
            gu += diff.sum(1)
            gv.index_add_(0, rows.reshape(-1), -diff.reshape(-1, diff.shape[2]))
    return loss, gx, gy
