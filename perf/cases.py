"""The work a user of this library has it do, as measurable cases.

Each case names a kind of call, its sizes and its options.  `listed()` gives
the cases that are always measured, `draw()` one more of the same ranges,
`prepare()` what a user's program holds before the call (inputs made from the
seed, resident graphs, weights), `run()` one pass through the public entry
points, `work()` the bytes and operations a pass cannot do without, and
`exact()` the same outputs from plain torch in 64 bits.

Graphs come from four seeded families, all made here with torch: uniform
random edges, R-MAT (0.57, 0.19, 0.19), a Chung-Lu power law (the degree law
of preferential attachment) and a block model.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "rust-igraph_b200"))

import igraph_b200 as ig  # noqa: E402
from igraph_b200 import warmstart  # noqa: E402

D = 0.85  # the reference's damping


# ------------------------------------------------------------------ the cases


def listed():
    return [
        # a small analysis graph through the one-call drop-in: the shape of the
        # reference's own micro-benchmark, G(1000, 0.05)
        {"name": "pagerank_er_1k", "kind": "pagerank", "n": 1000, "m": 25_000, "directed": False},
        # personalised ranks of a handful of vertices on a 10 k-vertex directed
        # graph, one call from host arrays
        {"name": "ppr_er_10k", "kind": "ppr", "n": 10_000, "m": 100_000, "seeds": 5, "directed": True},
        # weighted ranks of a mid-sized undirected graph, one call from host arrays
        {"name": "weighted_call_100k", "kind": "weighted_call", "n": 100_003, "m": 800_021, "directed": False},
        # the same on a resident graph of a million vertices, solved again and again
        {"name": "weighted_solve_1m", "kind": "weighted_solve", "n": 1_000_000, "m": 8_000_000, "directed": False},
        # the headline: FP32 matvecs, FP64 residuals, certified error, R-MAT scale 24
        {"name": "refined_rmat_s24", "kind": "refined", "scale": 24, "edge_factor": 16},
        # a graph that changes between solves: device edges -> CSR -> FP64 power
        # iteration with the reference's stop rule
        {"name": "build_solve_rmat_s22", "kind": "build_solve", "scale": 22, "edge_factor": 16},
        # a batch of personalised vectors on a community graph, ragged last tile
        {"name": "batch_sbm_1m", "kind": "batch", "n": 1_000_000, "m": 10_000_000, "blocks": 64, "columns": 200},
        # eigenvector centrality of an undirected graph, one call from host arrays
        {"name": "eigenvector_50k", "kind": "eigenvector", "n": 50_001, "m": 400_000},
        # hub and authority scores of a directed web-like graph, one call
        {"name": "hits_rmat_s19", "kind": "hits", "scale": 19, "edge_factor": 16},
        # an edge-list text to ranks through the linear-system solver
        {"name": "text_linsys_3m", "kind": "text", "n": 400_000, "m": 3_000_000},
        # inference of the learned start vector (shipped weights)
        {"name": "warm_predict_s22", "kind": "predict", "scale": 22, "edge_factor": 16},
        # loss and gradient of the warm-start network on a training graph
        {"name": "warm_grad_500k", "kind": "grad", "n": 500_009, "m": 3_000_000, "directed": True},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pagerank", "ppr", "weighted_call", "weighted_solve", "refined", "build_solve", "batch",
                       "eigenvector", "hits", "text", "predict", "grad"])
    c = {"kind": kind}
    if kind == "pagerank":
        n = _logint(rng, 34, 12_000)
        c.update(n=n, m=int(n * rng.uniform(2, 25)), directed=rng.random() < 0.5)
    elif kind == "ppr":
        n = _logint(rng, 500, 100_000)
        c.update(n=n, m=int(n * rng.uniform(3, 14)), seeds=_logint(rng, 1, 100), directed=rng.random() < 0.7)
    elif kind == "weighted_call":
        n = _logint(rng, 3_000, 300_000)
        c.update(n=n, m=int(n * rng.uniform(3, 10)), directed=rng.random() < 0.3)
    elif kind == "weighted_solve":
        n = _logint(rng, 100_000, 1_500_000)
        c.update(n=n, m=int(n * rng.uniform(4, 10)), directed=rng.random() < 0.3)
    elif kind == "refined":
        c.update(scale=rng.randint(19, 23), edge_factor=rng.randint(10, 18))
    elif kind == "build_solve":
        c.update(scale=rng.randint(18, 22), edge_factor=rng.randint(9, 17))
    elif kind == "batch":
        n = _logint(rng, 50_000, 1_000_000)
        c.update(n=n, m=int(n * rng.uniform(5, 10)), blocks=rng.choice([16, 32, 64]), columns=_logint(rng, 8, 190))
    elif kind == "eigenvector":
        n = _logint(rng, 2_000, 60_000)
        c.update(n=n, m=int(n * rng.uniform(4, 8)))
    elif kind == "hits":
        c.update(scale=rng.randint(14, 19), edge_factor=rng.randint(9, 17))
    elif kind == "text":
        n = _logint(rng, 20_000, 400_000)
        c.update(n=n, m=int(n * rng.uniform(3, 8)))
    elif kind == "predict":
        c.update(scale=rng.randint(18, 22), edge_factor=rng.randint(9, 17))
    else:
        n = _logint(rng, 100_000, 700_000)
        c.update(n=n, m=int(n * rng.uniform(4, 8)), directed=rng.random() < 0.5)
    return c


# ------------------------------------------------------------------ seeded inputs (torch)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform_edges(n, m, g):
    f = torch.randint(0, n, (m,), device="cuda", generator=g, dtype=torch.int32)
    t = torch.randint(0, n, (m,), device="cuda", generator=g, dtype=torch.int32)
    return f, t


def _rmat_edges(scale, m, g, a=0.57, b=0.19, c=0.19):
    f = torch.zeros(m, device="cuda", dtype=torch.int32)
    t = torch.zeros(m, device="cuda", dtype=torch.int32)
    for _ in range(scale):
        r = torch.rand(m, device="cuda", generator=g)
        down = r >= a + b
        right = ((r >= a) & (r < a + b)) | (r >= a + b + c)
        f.mul_(2).add_(down)
        t.mul_(2).add_(right)
    return f, t


def _powerlaw_edges(n, m, g, alpha=0.5, offset=8.0):
    w = (torch.arange(n, device="cuda", dtype=torch.float64) + offset).pow_(-alpha)
    cdf = torch.cumsum(w, 0)
    cdf /= cdf[-1].clone()

    def pick():
        r = torch.rand(m, device="cuda", generator=g, dtype=torch.float64)
        return torch.searchsorted(cdf, r).clamp_(max=n - 1).to(torch.int32)

    return pick(), pick()


def _block_edges(n, m, blocks, g, inside=0.8):
    size = n // blocks
    f = torch.randint(0, n, (m,), device="cuda", generator=g)
    stay = torch.rand(m, device="cuda", generator=g) < inside
    near = (f // size) * size + torch.randint(0, size, (m,), device="cuda", generator=g)
    far = torch.randint(0, n, (m,), device="cuda", generator=g)
    t = torch.where(stay, near.clamp_(max=n - 1), far)
    return f.to(torch.int32), t.to(torch.int32)


def _edges(case, seed):
    """(n, from, to) of a case as int32 CUDA tensors."""
    g = _gen(seed)
    kind = case["kind"]
    if "scale" in case:
        n = 1 << case["scale"]
        f, t = _rmat_edges(case["scale"], n * case["edge_factor"], g)
    elif kind in ("pagerank", "ppr"):
        n = case["n"]
        f, t = _uniform_edges(n, case["m"], g)
    elif kind == "batch":
        n = case["n"]
        f, t = _block_edges(n, case["m"], case["blocks"], g)
    else:
        n = case["n"]
        f, t = _powerlaw_edges(n, case["m"], g)
    if kind == "text":  # read_edgelist takes n from the largest id
        f[0] = n - 1
    return n, f, t


def _weights(case, seed):
    return 0.5 + 1.5 * torch.rand(case["m"], device="cuda", generator=_gen(seed + 7919), dtype=torch.float64)


def _seed_vertices(case, seed):
    return np.random.default_rng(seed).choice(case["n"], min(case["seeds"], case["n"]), replace=False).astype(np.uint32)


def _seed_lists(case, seed):
    """1 to 1000 seeds a column, log-uniform."""
    r = np.random.default_rng(seed)
    return [r.integers(0, case["n"], int(math.exp(r.uniform(0.0, math.log(1000.0))))).astype(np.uint32)
            for _ in range(case["columns"])]


def _text(f, t):
    """The edges as "u v" lines without leading zeros, as bytes."""
    m = len(f)
    width = 7
    a = np.empty((m, 2 * width + 2), np.uint8)
    keep = np.ones(a.shape, bool)
    for off, v in ((0, f), (width + 1, t)):
        v = v.astype(np.int64)
        for k in range(width):
            p = 10 ** (width - 1 - k)
            a[:, off + k] = 48 + (v // p) % 10
            if k < width - 1:
                keep[:, off + k] = v >= p
    a[:, width] = 32
    a[:, -1] = 10
    return a[keep].tobytes()


PARAMS = {"W1": (32, 16), "b1": (32,), "Wm1": (8, 32), "W2": (32, 48), "b2": (32,), "Wm2": (8, 32), "W3": (8, 48),
          "b3": (8,)}  # the network's parameters in their order in memory


def _network(case, seed):
    """The shipped weights for inference, a fresh initialisation for training."""
    if case["kind"] == "predict":
        with open(os.path.join(ROOT, "rust-igraph_b200", "igraph_b200", "warmstart_weights.f32"), "rb") as fh:
            return np.frombuffer(fh.read()[12:], np.float32).copy()
    r = np.random.default_rng(seed + 5)
    parts = []
    for name, shape in PARAMS.items():
        if len(shape) == 1:
            p = np.zeros(shape) if name == "b3" else np.full(shape, 0.05)
        else:
            p = r.uniform(-1.0, 1.0, shape) * math.sqrt(6.0 / shape[1])
            if name == "W3":
                p[1:] = 0.0
        parts.append(p.ravel())
    return np.concatenate(parts).astype(np.float32)


def _host(x):
    return x.cpu().numpy().view(np.uint32)


# ------------------------------------------------------------------ prepare and run


def prepare(case, seed):
    kind = case["kind"]
    n, f, t = _edges(case, seed)
    s = {"kind": kind, "n": n}
    torch.cuda.synchronize()
    if kind in ("pagerank", "ppr", "weighted_call", "eigenvector", "hits"):
        directed = True if kind == "hits" else case.get("directed", False)
        s["graph"] = ig.Graph.from_edge_arrays(n, _host(f), _host(t), directed)
        if kind == "ppr":
            s["vids"] = _seed_vertices(case, seed)
        if kind == "weighted_call":
            s["weights"] = _weights(case, seed).cpu().numpy()
        return s
    if kind == "text":
        s["text"] = _text(_host(f), _host(t))
        s["out"] = torch.empty(n, dtype=torch.float64, device="cuda")
        return s
    if kind == "build_solve":
        s.update(f=f, t=t, out=torch.empty(n, dtype=torch.float64, device="cuda"))
        return s
    w = None
    if kind == "weighted_solve":
        w = _weights(case, seed)
        torch.cuda.synchronize()
    s["dg"] = ig.DeviceGraph.from_device(n, f.numel(), f.data_ptr(), t.data_ptr(), _directed(case),
                                         w.data_ptr() if w is not None else 0)
    if kind == "batch":
        s["lists"] = _seed_lists(case, seed)
        s["out"] = torch.empty((n, case["columns"]), dtype=torch.float32, device="cuda")
        return s
    s["out"] = torch.empty(n, dtype=torch.float64, device="cuda")
    if kind in ("predict", "grad"):
        s["net"] = warmstart.WarmStartNet(1)
        s["net"].set_params(_network(case, seed))
    if kind == "grad":
        s["target"] = _pagerank(_arcs(n, f, t, case["directed"]), stop=1e-12)
        torch.cuda.synchronize()
    return s


def _directed(case):
    return case.get("directed", case["kind"] != "batch")


def run(s):
    kind = s["kind"]
    if kind == "pagerank":
        return ig.pagerank(s["graph"])
    if kind == "ppr":
        return ig.personalized_pagerank_vs(s["graph"], s["vids"], D)
    if kind == "weighted_call":
        return ig.pagerank_weighted(s["graph"], s["weights"])
    if kind == "weighted_solve":
        s["dg"].solve_device(s["out"].data_ptr())
        return s["out"]
    if kind == "refined":
        s["dg"].solve_device(s["out"].data_ptr(), ig.Options(precision=ig.PRECISION_FP32_REFINED))
        return s["out"]
    if kind == "build_solve":
        with ig.DeviceGraph.from_device(s["n"], s["f"].numel(), s["f"].data_ptr(), s["t"].data_ptr(), True) as dg:
            dg.solve_device(s["out"].data_ptr())
        return s["out"]
    if kind == "batch":
        s["dg"].ppr_batch(s["lists"], D, 1e-8, d_out=s["out"].data_ptr())
        return s["out"]
    if kind == "eigenvector":
        return list(ig.eigenvector_centrality(s["graph"], with_eigenvalue=True))
    if kind == "hits":
        r = ig.hub_and_authority_scores(s["graph"])
        return {"hub": r.hub, "authority": r.authority, "eigenvalue": r.eigenvalue}
    if kind == "text":
        with ig.DeviceGraph.from_edgelist(s["text"]) as dg:
            dg.solve_device(s["out"].data_ptr(), ig.Options(precision=ig.PRECISION_LINSYS))
        return s["out"]
    if kind == "predict":
        s["net"].predict(s["dg"], s["out"].data_ptr())
        return s["out"]
    loss, grad = s["net"].loss_grad(s["dg"], s["target"].data_ptr())
    return {"loss": loss, "grad": grad}


# ------------------------------------------------------------------ what a pass cannot do without

# Applications of the graph's operator that reach each call's tolerance on
# these families (about what the reference's rules take; the Krylov counts are
# the matvecs of the two-term methods).  The eigenvector rule, a change below
# 1e-14, lies under the rounding of such vectors, so it runs to its cap of 5000.
APPLICATIONS = {"pagerank": 20, "ppr": 20, "weighted_call": 22, "weighted_solve": 22, "refined": 14,
                "build_solve": 28, "batch": 24, "eigenvector": 5000, "hits": 30, "text": 24, "predict": 2, "grad": 4}


def work(case):
    kind = case["kind"]
    n = 1 << case["scale"] if "scale" in case else case["n"]
    m = n * case["edge_factor"] if "scale" in case else case["m"]
    arcs = m if (True if kind == "hits" else _directed(case) and kind not in ("text", "eigenvector")) else 2 * m
    k = APPLICATIONS[kind]
    width = {"refined": 4, "predict": 32, "grad": 32}.get(kind, 8)  # bytes of a vertex's value
    cols = case.get("columns", 1)
    if kind == "batch":
        width = 4 * cols
    # the index stream (and weights) and one read and one write of the vertex values per application
    per = 4.0 * arcs + (8.0 * arcs if kind.startswith("weighted") else 0.0) + 4.0 * n + 2.0 * width * n
    if kind == "hits":
        per += 4.0 * arcs
    io = 8.0 * m if kind in ("pagerank", "ppr", "weighted_call", "eigenvector", "hits", "build_solve") else 0.0
    if kind == "text":
        io = 13.0 * m
    flops = 2.0 * arcs * k * (8 if kind in ("predict", "grad") else cols)
    if kind in ("predict", "grad"):
        flops += 2.0 * n * 2600 * (3 if kind == "grad" else 1)
    return {"bytes": k * per + io + (4.0 * cols if kind == "batch" else 8.0) * n, "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits, plain torch


class _Arcs:
    """In-arc matrix A[v, u] = sum of the weights of arcs u -> v, and the out-strengths."""

    def __init__(self, n, src, dst, w):
        self.n = n
        order = torch.argsort(dst, stable=True)
        crow = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        crow[1:] = torch.cumsum(torch.bincount(dst, minlength=n), 0)
        self.indeg = crow[1:] - crow[:-1]
        val = torch.ones(len(src), dtype=torch.float64, device="cuda") if w is None else w
        self.a = torch.sparse_csr_tensor(crow, src[order].to(torch.int64), val[order], (n, n))
        self.outdeg = torch.bincount(src, minlength=n)
        self.out = self.outdeg.to(torch.float64) if w is None else torch.bincount(src, weights=w, minlength=n)

    def mul(self, x):
        return self.a @ x


def _arcs(n, f, t, directed, w=None, reverse=False):
    if not directed:
        f, t = torch.cat([f, t]), torch.cat([t, f])
        w = None if w is None else torch.cat([w, w])
    return _Arcs(n, t, f, w) if reverse else _Arcs(n, f, t, w)


def _pagerank(a, reset=None, stop=1e-10, most=1000):
    """The damped power iteration to a successive L1 change below `stop` (columns of `reset` together)."""
    n = a.n
    x = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda") if reset is None else reset.clone()
    live = a.out > 0
    inv = torch.where(live, 1.0 / a.out.clamp(min=1e-300), torch.zeros_like(a.out))
    if x.dim() == 2:
        inv, live = inv[:, None], live[:, None]
    for _ in range(most):
        lost = (x * ~live).sum(0)
        g = a.mul(x * inv)
        if reset is None:
            y = (1.0 - D) / n + D * lost / n + D * g
        else:
            y = (1.0 - D) * reset + D * (g + lost * reset)
        change = float((y - x).abs().sum(0).max())
        x = y
        if change < stop:
            break
    return x


def _seed_columns(n, lists):
    r = torch.zeros((n, len(lists)), dtype=torch.float64, device="cuda")
    for k, v in enumerate(lists):
        i = torch.as_tensor(v.astype(np.int64), device="cuda")
        r[:, k].index_add_(0, i, torch.full((len(v),), 1.0 / len(v), dtype=torch.float64, device="cuda"))
    return r


def _bf16(x):
    return x.to(torch.bfloat16).to(torch.float64)


def _slog(z):
    return torch.sign(z) * torch.log1p(z.abs())


def _forward(params, a):
    """The warm-start network with its 16-bit operands, all sums in 64 bits."""
    p, at = {}, 0
    flat = torch.as_tensor(params, device="cuda").to(torch.float64)
    for name, shape in PARAMS.items():
        size = int(np.prod(shape))
        p[name] = flat[at:at + size].reshape(shape)
        at += size
    n = a.n
    li, lo = torch.log1p(a.indeg.double()), torch.log1p(a.outdeg.double())
    x0 = torch.zeros((n, 16), dtype=torch.float64, device="cuda")
    x0[:, 0], x0[:, 1], x0[:, 2], x0[:, 3] = li / 8, lo / 8, (a.outdeg == 0).double(), 1.0
    x0[:, 4], x0[:, 5] = (li - lo) / 8, math.log(n) / 16
    x0 = _bf16(x0)
    sc = torch.where(a.outdeg > 0, 1.0 / a.outdeg.clamp(min=1).double(), torch.zeros_like(a.out))[:, None]
    h0 = _bf16((x0 @ _bf16(p["W1"]).T + p["b1"]).clamp_(min=0.0))
    s1 = a.mul((h0 @ _bf16(p["Wm1"]).T) * sc)
    z1 = torch.cat([h0, _bf16(_slog(s1)), torch.zeros((n, 8), dtype=torch.float64, device="cuda")], 1)
    h1 = _bf16((z1 @ _bf16(p["W2"]).T + p["b2"]).clamp_(min=0.0))
    s2 = a.mul((h1 @ _bf16(p["Wm2"]).T) * sc)
    z2 = torch.cat([h1, _bf16(_slog(s2)), torch.zeros((n, 8), dtype=torch.float64, device="cuda")], 1)
    y = z2 @ _bf16(p["W3"][0]) + p["b3"][0]
    return p, sc, x0, h0, z1, s1, h1, z2, s2, y


def _gradient(params, a, back, target):
    n = a.n
    p, sc, x0, h0, z1, s1, h1, z2, s2, y = _forward(params, a)
    tv = target.clamp(min=1e-300)
    w = n * tv
    e = y - torch.log(w)
    dy = 2.0 * w * e / n
    w3 = torch.zeros((8, 48), dtype=torch.float64, device="cuda")
    w3[0] = dy @ z2
    b3 = torch.zeros(8, dtype=torch.float64, device="cuda")
    b3[0] = dy.sum()
    g1 = back.mul(dy[:, None] * p["W3"][0, 32:40] / (1.0 + s2.abs())) * sc
    d1 = (dy[:, None] * p["W3"][0, :32] + g1 @ p["Wm2"]) * (h1 > 0)
    dz = d1 @ p["W2"]
    g0 = back.mul(dz[:, 32:40] / (1.0 + s1.abs())) * sc
    d0 = (dz[:, :32] + g0 @ p["Wm1"]) * (h0 > 0)
    grad = torch.cat([(d0.T @ x0).ravel(), d0.sum(0), (g0.T @ h0).ravel(), (d1.T @ z1).ravel(), d1.sum(0),
                      (g1.T @ h1).ravel(), w3.ravel(), b3])
    return {"loss": float((w * e * e).sum() / n), "grad": grad.cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    n, f, t = _edges(case, seed)
    directed = True if kind == "hits" else _directed(case) and kind not in ("text", "eigenvector")
    if kind == "hits":
        a, b = _arcs(n, f, t, True), _arcs(n, f, t, True, reverse=True)
        h = a.out / a.out.max()
        lam = 0.0
        for _ in range(5000):
            y = b.mul(a.mul(h))
            top = float(y.abs().max())
            y = y / top if top > 0.0 else y
            lam = top if top > 0.0 else lam
            change = float((y - h).abs().sum())
            h = y
            if change < 1e-12:
                break
        au = a.mul(h)
        return {"hub": h.cpu().numpy(), "authority": (au / au.abs().max()).cpu().numpy(), "eigenvalue": lam}
    w = _weights(case, seed) if kind.startswith("weighted") else None
    a = _arcs(n, f, t, directed, w)
    if kind in ("pagerank", "weighted_call"):
        return _pagerank(a).cpu().numpy()
    if kind == "ppr":
        return _pagerank(a, _seed_columns(n, [_seed_vertices(case, seed)])[:, 0]).cpu().numpy()
    if kind in ("weighted_solve", "build_solve"):
        return _pagerank(a)
    if kind in ("refined", "text"):
        x = _pagerank(a, stop=1e-15, most=300)
        return x / x.sum() if kind == "refined" else x
    if kind == "batch":
        return _pagerank(a, _seed_columns(n, _seed_lists(case, seed)), stop=1e-13, most=250)
    if kind == "eigenvector":
        x = torch.ones(n, dtype=torch.float64, device="cuda")
        for _ in range(5000):
            y = x + a.mul(x)
            y /= y.abs().max()
            change = float((y - x).abs().sum())
            x = y
            if change < 1e-14:
                break
        lam = float((x @ a.mul(x)) / (x @ x))
        return [x.cpu().numpy(), lam]
    if kind == "predict":
        y = _forward(_network(case, seed), a)[-1]
        e = torch.exp(y - y.max())
        return e / e.sum()
    back = _arcs(n, f, t, directed, reverse=True)
    return _gradient(_network(case, seed), a, back, _pagerank(a, stop=1e-12))
