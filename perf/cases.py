"""What this framework is measured on: the applications a user runs on a graph
handle, through the package's public functions.

The graphs are the repository's own synthetic ones, drawn here with torch from
the seed alone: R-MAT (a, b, c, d = .57, .19, .19, .05, self loops and
duplicates removed, sorted by source; ids at or above n dropped where n is not
a power of two), directed or symmetrised, and the batch of independent
Erdos-Renyi graphs.  A state is what a program keeps between calls: the graph
handle with its weights, the sources or seeds, the input vectors on the GPU.
"""
import math

import numpy as np
import torch

import polymer_b200 as pm

DEV = "cuda"
DAMPING = 0.85
PSI = ((0.9, 0.1), (0.1, 0.9))
VALUE = ("pagerank", "spmv", "bp")
TRAVERSAL = ("bfs", "cc", "bf", "cc_bf", "trio")


def listed():
    return [
        # a small analysis, run often: ten iterations in the reference's own precision on 2^16 vertices
        dict(name="pagerank-f64-64k", kind="pagerank", n=1 << 16, ef=16, sym=False, iters=10, dtype="f64"),
        # the value applications at scale: a crawl-sized graph whose ids alone are larger than L2
        dict(name="pagerank-f32-16m", kind="pagerank", n=1 << 24, ef=16, sym=False, iters=20, dtype="f32"),
        dict(name="spmv-f32-16m", kind="spmv", n=1 << 24, ef=16, sym=False, iters=10, dtype="f32"),
        dict(name="bp-f32-16m", kind="bp", n=1 << 24, ef=16, sym=False, iters=10, dtype="f32"),
        # queries on a small undirected graph of odd size, where launches and round trips count
        dict(name="trio-10k", kind="trio", n=10007, ef=8, sym=True, sources=1),
        # traversals of a social-network-sized undirected graph
        dict(name="bfs-16-sources-4m", kind="bfs", n=1 << 22, ef=16, sym=True, sources=16),
        dict(name="components-bellman-4m", kind="cc_bf", n=1 << 22, ef=16, sym=True, sources=1),
        # batched queries: 64 sources in one traversal; 50 shortest-path sources on a ragged graph; 32 personalised vectors
        dict(name="bfs-64-lanes-4m", kind="bfs_multi", n=1 << 22, ef=16, sym=True, sources=64),
        dict(name="bellman-50-lanes-1500007", kind="bf_multi", n=1500007, ef=16, sym=True, sources=50),
        dict(name="ppr-32-seeds-16m", kind="ppr", n=1 << 24, ef=16, sym=False, iters=20, sources=32),
        # many small graphs of uneven size in one call
        dict(name="parts-256", kind="parts", count=256, n_min=1000, n_max=100000, ef=8, iters=20),
        # learning edge weights: the weighted fixed point, its adjoint, and one weighted product's backward
        dict(name="train-1m", kind="train", n=1 << 20, ef=16, sym=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same kinds; sizes over the logarithm of the whole range, mostly not powers of two."""
    kind = rng.choice(VALUE + VALUE + TRAVERSAL + ("bfs_multi", "bf_multi", "ppr", "parts", "train"))
    ef = rng.choice((4, 8, 12, 16))
    if kind in VALUE:
        return dict(kind=kind, n=_log_int(rng, 1 << 10, 1 << 24), ef=ef, sym=rng.random() < 0.25 and kind != "spmv",
                    iters=rng.randint(5, 20), dtype=rng.choice(("f32", "f32", "f64")))
    if kind in TRAVERSAL:
        return dict(kind=kind, n=_log_int(rng, 1 << 10, 1 << 22), ef=ef, sym=rng.random() < 0.75,
                    sources=rng.randint(1, 16) if kind == "bfs" else 1)
    if kind == "bfs_multi":
        return dict(kind=kind, n=_log_int(rng, 1 << 10, 1 << 22), ef=ef, sym=rng.random() < 0.75, sources=rng.randint(2, 64))
    if kind == "bf_multi":
        return dict(kind=kind, n=_log_int(rng, 1 << 10, 1 << 21), ef=ef, sym=rng.random() < 0.75, sources=rng.randint(2, 64))
    if kind == "ppr":
        return dict(kind=kind, n=_log_int(rng, 1 << 10, 1 << 23), ef=ef, sym=False, iters=rng.randint(5, 20),
                    sources=rng.randint(1, 32))
    if kind == "parts":
        n_min = _log_int(rng, 100, 5000)
        return dict(kind=kind, count=_log_int(rng, 8, 400), n_min=n_min, n_max=n_min * rng.randint(2, 20), ef=rng.choice((4, 8)),
                    iters=rng.randint(5, 20))
    return dict(kind="train", n=_log_int(rng, 1 << 10, 1 << 21), ef=ef, sym=False)


# ---- inputs -----------------------------------------------------------------
def _csr(keys, n):
    """(offsets, ids) of sorted unique (src << 32 | dst) keys."""
    off = torch.searchsorted(keys, torch.arange(n + 1, device=DEV, dtype=torch.int64) << 32).to(torch.int32)
    return off, (keys & 0xFFFFFFFF).to(torch.int32)


def _unique(keys):
    keys = torch.sort(keys).values
    keep = torch.ones(keys.numel(), dtype=torch.bool, device=DEV)
    keep[1:] = keys[1:] != keys[:-1]
    return keys[keep]


def _rmat(n, ef, sym, gen, edges=None):
    """R-MAT of n * ef draws; with edges, exactly that many distinct ones, picked from three times as many draws."""
    draws = n * ef if edges is None else 3 * edges
    s = torch.zeros(draws, dtype=torch.int64, device=DEV)
    d = torch.zeros(draws, dtype=torch.int64, device=DEV)
    for _ in range(max(1, (n - 1).bit_length())):
        u = torch.rand(draws, device=DEV, generator=gen)
        s.mul_(2).add_(u >= 0.76)
        d.mul_(2).add_(((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    keep = (s != d) & (s < n) & (d < n)
    s, d = s[keep], d[keep]
    keys = (s << 32) | d
    if sym:
        keys = torch.cat([keys, (d << 32) | s])
    keys = _unique(keys)
    if edges is not None:
        keys = torch.sort(keys[torch.randperm(keys.numel(), device=DEV, generator=gen)[:edges]]).values
    return _csr(keys, n)


def _er(case, gen):
    """(offsets, ids, first vertex of each part) of independent directed Erdos-Renyi graphs."""
    u = np.random.RandomState(case["count"]).uniform(size=case["count"])  # the sizes belong to the case
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    sizes = np.floor(np.exp(lo + u * (hi - lo))).astype(np.int64).clip(case["n_min"], case["n_max"])
    base = np.concatenate([[0], np.cumsum(sizes)])
    first = torch.from_numpy(base[:-1]).to(DEV)
    size = torch.from_numpy(sizes).to(DEV)
    part = torch.repeat_interleave(torch.arange(case["count"], device=DEV), size * case["ef"])
    s = first[part] + (torch.rand(part.numel(), device=DEV, generator=gen, dtype=torch.float64) * size[part]).long()
    d = first[part] + (torch.rand(part.numel(), device=DEV, generator=gen, dtype=torch.float64) * size[part]).long()
    keep = s != d
    return (*_csr(_unique((s[keep] << 32) | d[keep]), int(base[-1])), base)


def _inputs(case, seed):
    """Every input of a case, from the seed alone: plain tensors and arrays."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    kind = case["kind"]
    x = {"kind": kind}
    if kind == "parts":
        x["off"], x["idx"], x["base"] = _er(case, gen)
        return x
    n = case["n"]
    # a training case's gradients are per edge: its edge count is the case's
    x["off"], x["idx"] = _rmat(n, case["ef"], case["sym"], gen, n * case["ef"] if kind == "train" else None)
    m = x["idx"].numel()
    deg = (x["off"][1:] - x["off"][:-1]).long()
    f = torch.float64 if case.get("dtype") == "f64" else torch.float32
    if kind == "spmv":
        x["w"] = 1.0 - torch.rand(m, device=DEV, generator=gen)
        x["x0"] = torch.rand(n, device=DEV, generator=gen).to(f)
    if kind == "bp":
        x["prior"] = torch.rand((n, 2), device=DEV, generator=gen).clamp_(1e-6, 1 - 1e-6).to(f)
    if kind == "train":
        w = torch.randn(m, device=DEV, generator=gen).exp_()
        row = torch.repeat_interleave(torch.arange(n, device=DEV), deg)
        total = torch.zeros(n, device=DEV, dtype=torch.float64).index_add_(0, row, w.double())
        x["w"] = (w.double() / total[row]).float()
        x["grad_p"] = torch.zeros(n, device=DEV)
        x["grad_p"][torch.randint(0, n, (min(1024, n),), device=DEV, generator=gen)] = 1.0
        x["x"] = torch.rand(n, device=DEV, generator=gen)
        x["grad_y"] = torch.rand(n, device=DEV, generator=gen)
    if kind in ("bf", "cc_bf", "trio", "bf_multi"):  # int weights in [1, 22], the same in both directions
        row = torch.repeat_interleave(torch.arange(n, device=DEV), deg)
        col = x["idx"].long()
        a, b = torch.minimum(row, col), torch.maximum(row, col)
        h = (a * 0x9E3779B1 + b * 0x85EBCA77 + seed * 0xC2B2AE3D) & 0xFFFFFFFFFFFF
        h = ((h ^ (h >> 21)) * 0x27D4EB2F) & 0xFFFFFFFFFFFF
        x["w"] = (1 + ((h >> 13) % 22)).to(torch.int32)
    if "sources" in case:  # vertices with out-edges
        have = torch.nonzero(deg > 0).flatten()
        pick = torch.randint(0, have.numel(), (case["sources"],), device=DEV, generator=gen)
        x["sources"] = have[pick].to(torch.int32).cpu().numpy()
    return x


def prepare(case, seed):
    x = _inputs(case, seed)
    torch.cuda.synchronize()
    x["g"] = pm.Graph.from_csr(x.pop("off"), x.pop("idx"), symmetric=bool(case.get("sym")), weights=x.pop("w", None))
    if "base" in x:
        x["g"].set_parts(x.pop("base"))
    x["iters"] = case.get("iters", 0)
    x["dtype"] = np.float64 if case.get("dtype") == "f64" else np.float32
    x["like"] = torch.empty(1, device=DEV)  # results stay on the GPU
    return x


def run(state):
    g, like, kind, iters = state["g"], state["like"], state["kind"], state["iters"]
    if kind == "pagerank":
        return pm.PageRank(g, iters, DAMPING, dtype=state["dtype"], device_out=like)
    if kind == "spmv":
        return pm.SPMV(g, state["x0"], iters, dtype=state["dtype"])
    if kind == "bp":
        return pm.BeliefPropagation(g, state["prior"], iters, PSI, dtype=state["dtype"])
    if kind == "bfs":  # depths; which of several parents one level up a vertex gets is not determined
        return [pm.BFS(int(s), g, device_out=like)[1] for s in state["sources"]]
    if kind == "cc":
        return pm.Components(g, device_out=like)
    if kind == "bf":
        return pm.BellmanFord(g, int(state["sources"][0]), device_out=like)
    if kind == "cc_bf":
        return pm.Components(g, device_out=like), pm.BellmanFord(g, int(state["sources"][0]), device_out=like)
    if kind == "trio":
        s = int(state["sources"][0])
        return pm.BFS(s, g, device_out=like)[1], pm.Components(g, device_out=like), pm.BellmanFord(g, s, device_out=like)
    if kind == "bfs_multi":
        return pm.BFSMulti(state["sources"], g, device_out=like)
    if kind == "bf_multi":
        return pm.BellmanFordMulti(state["sources"], g, device_out=like)
    if kind == "ppr":
        return pm.PersonalizedPageRank(g, state["sources"], iters, DAMPING, device_out=like)
    if kind == "parts":
        return pm.PageRankParts(g, iters, DAMPING, device_out=like)
    p, _, _ = pm.WeightedPageRank(g, DAMPING, 1e-6, device_out=like)
    dw, lam, _ = pm.PageRankAdjoint(g, p, state["grad_p"], DAMPING, 1e-6, with_lambda=True)
    dx, dw_y = pm.SpMVBackward(g, state["x"], state["grad_y"])
    return p, dw, lam, dx, dw_y


# ---- what a pass cannot do without -----------------------------------------
def work(case):
    """Bytes: every iteration of a value application reads the graph and its vector and writes the next one (the graph
    does not fit on the chip); a traversal reads the graph once and writes its results once."""
    kind = case["kind"]
    if kind == "parts":
        n = case["count"] * (case["n_max"] - case["n_min"]) / max(1e-9, math.log(case["n_max"] / case["n_min"]))
        m, it = n * case["ef"], case["iters"]
        return {"bytes": it * (4 * m + 16 * n), "flops": it * m}
    n = case["n"]
    m = n * case["ef"] * (1.9 if case["sym"] else 0.98) * (0.9 if n & (n - 1) else 1.0)
    v = 8 if case.get("dtype") == "f64" else 4
    it, k = case.get("iters", 1), case.get("sources", 1)
    if kind == "pagerank":
        return {"bytes": it * (4 * m + (4 + 3 * v) * n), "flops": it * m}
    if kind == "spmv":
        return {"bytes": it * (8 * m + (4 + 2 * v) * n), "flops": it * 2 * m}
    if kind == "bp":  # the counts of messages come from the graph once; every iteration updates the log-products
        return {"bytes": 4 * m + it * 8 * v * n, "flops": it * 12 * n}
    if kind == "bfs":  # each direction-optimised search touches a part of the edges; its results are written in full
        return {"bytes": k * (0.25 * m + 16 * n), "flops": 0}
    if kind == "cc":
        return {"bytes": 16 * n, "flops": 0}
    if kind == "bf":
        return {"bytes": 8 * m + 12 * n, "flops": m}
    if kind == "cc_bf":
        return {"bytes": 8 * m + 28 * n, "flops": m}
    if kind == "trio":
        return {"bytes": 8.25 * m + 44 * n, "flops": m}
    if kind == "bfs_multi":
        return {"bytes": 4 * m + (24 + 4 * k) * n, "flops": 0}
    if kind == "bf_multi":
        return {"bytes": 8 * m + (24 + 8 * k) * n, "flops": m * k}
    if kind == "ppr":
        return {"bytes": it * (4 * m + 8 * k * n), "flops": it * m * k}
    # 1e-6 takes about 55 passes forward and 70 back; then the weight gradients
    return {"bytes": 125 * (8 * m + 16 * n) + 2 * 12 * m + 8 * m, "flops": 125 * 2 * m}


# ---- the same results in 64 bits, with torch alone -----------------------------
def _matrix(rows, cols, vals, n):
    """CSR matrix with entries (rows, cols); rows need not be sorted."""
    order = torch.argsort(rows, stable=True)
    off = torch.searchsorted(rows[order], torch.arange(n + 1, device=DEV))
    return torch.sparse_csr_tensor(off, cols[order], vals[order], size=(n, n))


def _frontier_pagerank(pull, n, deg, iters, p0, added):
    p, q = p0.clone(), torch.zeros_like(p0)
    front = torch.ones(n, dtype=torch.bool, device=DEV)
    for _ in range(iters):
        c = torch.where(front & (deg > 0), p / deg.clamp(min=1), 0.0)
        both = pull @ torch.stack([c, front.double()], 1)
        q = q + both[:, 0]
        q = torch.where(front, DAMPING * q + added, q)
        p = torch.where(front, 0.0, p)
        p, q, front = q, p, both[:, 1] > 0.5
    return p


def _to_tol(step, x, tol, most=1000):
    for _ in range(most):
        y = step(x)
        rel = float((y - x).abs().sum() / y.abs().sum())
        x = y
        if rel <= tol:
            break
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind not in VALUE + ("ppr", "parts", "train"):
        return None  # integers: the same whatever computes them
    x = _inputs(case, seed)
    off, col = x["off"].long(), x["idx"].long()
    n, m = off.numel() - 1, col.numel()
    deg = off[1:] - off[:-1]
    row = torch.repeat_interleave(torch.arange(n, device=DEV), deg)
    if kind == "train":
        w = x["w"].double()
        fwd, back = _matrix(col, row, w, n), torch.sparse_csr_tensor(off, col, w, size=(n, n))
        p = _to_tol(lambda v: DAMPING * (fwd @ v[:, None])[:, 0] + (1 - DAMPING) / n,
                    torch.full((n,), 1.0 / n, device=DEV, dtype=torch.float64), 1e-6)
        gp = x["grad_p"].double()
        lam = _to_tol(lambda v: DAMPING * (back @ v[:, None])[:, 0] + gp, gp, 1e-6)
        gy = x["grad_y"].double()
        return p, DAMPING * lam[col] * p[row], lam, (back @ gy[:, None])[:, 0], gy[col] * x["x"].double()[row]
    w = x["w"].double() if kind == "spmv" else torch.ones(m, device=DEV, dtype=torch.float64)
    pull = _matrix(col, row, w, n)
    del row, col, w
    if kind == "spmv":
        v = x["x0"].double()
        for _ in range(case["iters"]):
            v = (pull @ v[:, None])[:, 0]
        return v
    if kind == "pagerank":
        p0 = torch.full((n,), 1.0 / n, device=DEV, dtype=torch.float64)
        return _frontier_pagerank(pull, n, deg, case["iters"], p0, (1 - DAMPING) / n)
    if kind == "parts":
        size = np.diff(x["base"])
        p0 = torch.from_numpy(np.repeat(1.0 / size, size)).to(DEV)
        return _frontier_pagerank(pull, n, deg, case["iters"], p0, (1 - DAMPING) * p0)
    if kind == "ppr":
        k = case["sources"]
        seeds = torch.from_numpy(x["sources"]).long().to(DEV)
        y = torch.zeros((n, k), device=DEV, dtype=torch.float64)
        y[seeds, torch.arange(k, device=DEV)] = 1.0
        for _ in range(case["iters"]):
            y = DAMPING * (pull @ (y / deg.clamp(min=1)[:, None] * (deg > 0)[:, None]))
            y[seeds, torch.arange(k, device=DEV)] += 1 - DAMPING
        return y
    # belief propagation: log-products, messages normalised to sum 1
    prior, psi = x["prior"].double(), torch.tensor(PSI, device=DEV, dtype=torch.float64)
    a, b = torch.zeros((n, 2), device=DEV, dtype=torch.float64), torch.zeros((n, 2), device=DEV, dtype=torch.float64)
    front = torch.ones(n, dtype=torch.bool, device=DEV)
    for _ in range(case["iters"]):
        k = (pull @ front.double()[:, None])
        e = prior * torch.exp(a - a.max(1, keepdim=True).values)
        msg = e @ psi.T
        b = torch.where(front[:, None], 0.0, b) + k * (torch.log(msg) - torch.log(msg.sum(1, keepdim=True)))
        a, b, front = b, a, k[:, 0] > 0
    return a
