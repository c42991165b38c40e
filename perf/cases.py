"""Workloads of the PageRank library, through its public Python entry points.

Graph shapes are those of the repository's benchmark and tests: R-MAT graphs
(16 draws a vertex, a/b/c 0.57/0.19/0.19), web-like graphs (Zipf out-degrees,
70% of the targets near their source, 38 edges a vertex) and square grids with
a few diagonals.  They are drawn on the GPU from the seed, self-loops are added
by the library, and the solves use the library's default options unless the
case says otherwise.

Kinds of work:
  static   prx_solve of a whole graph from uniform ranks (FP64, the reference's
           drop-in), or with `refine` on FP32 storage with FP64 refinement
  dynamic  ND / DT / DF / DF-P from the previous ranks on an updated graph
  update   what a serving loop does with a raw batch: tidy it, apply it on the
           device, DF-P from the previous ranks, and roll the batch back
  ppr      batched personalized PageRank of up to 64 teleport sets
  adjoint  a training step: weights in, ranks, and gradients of a loss
  ingest   an edge list already on the GPU -> graph -> ranks
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(1, os.path.join(ROOT, "pagerank-cuda-dynamic_gb300"))
import pagerank_gb300 as pg  # noqa: E402

DEV = "cuda"
ALPHA, TOL, CAP = 0.85, 1e-10, 500
MODES = {"nd": "NAIVE_DYNAMIC", "dt": "DYNAMIC_TRAVERSAL", "df": "DYNAMIC_FRONTIER", "dfp": "PRUNE_DYNAMIC_FRONTIER"}
_ctx = []


def ctx():
    """One context for the process, as a program keeps it."""
    if not _ctx:
        _ctx.append(pg.Context(0))
    return _ctx[0]


# ---- the cases -------------------------------------------------------------------
def listed():
    return [
        # a small graph solved from a service: launches and the host path count
        {"name": "static_rmat10", "kind": "static", "graph": "rmat", "n": 1 << 10, "refine": False},
        # the benchmark's R-MAT graph of scale 16: everything stays in L2
        {"name": "static_rmat16", "kind": "static", "graph": "rmat", "n": 1 << 16, "refine": False},
        # a road-like graph: in-degrees of 5 to 7, high diameter
        {"name": "static_grid4096", "kind": "static", "graph": "grid", "n": 4096 * 4096, "refine": False},
        # a web crawl, the benchmark's headline shape
        {"name": "static_web20m", "kind": "static", "graph": "web", "n": 20_000_003, "refine": False},
        # a web crawl on FP32 storage with FP64 refinement
        {"name": "refine_web6m", "kind": "static", "graph": "web", "n": 6_000_001, "refine": True},
        # new ranks after a few edges changed, the graph already updated
        {"name": "df_rmat18", "kind": "dynamic", "graph": "rmat", "n": 1 << 18, "mode": "df", "batch": 400},
        # reachability marking on a high-diameter graph
        {"name": "dt_grid1000", "kind": "dynamic", "graph": "grid", "n": 1000 * 1000, "mode": "dt", "batch": 512},
        # a serving loop's update of a web-like graph, 1e-4 of its edges
        {"name": "update_web3m", "kind": "update", "graph": "web", "n": 3_000_017, "batch": 11_400},
        # a full block of personalized vectors on FP32 storage
        {"name": "ppr32_rmat20", "kind": "ppr", "graph": "rmat", "n": 1 << 20, "vectors": 64, "refine": True},
        # some personalized vectors in FP64
        {"name": "ppr64_web200k", "kind": "ppr", "graph": "web", "n": 200_003, "vectors": 24, "refine": False},
        # a training step over edge weights
        {"name": "adjoint_rmat18", "kind": "adjoint", "graph": "rmat", "n": 1 << 18},
        # a new edge list ranked once
        {"name": "ingest_web3m", "kind": "ingest", "graph": "web", "n": 3_000_001},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["static", "static", "dynamic", "update", "ppr", "adjoint", "ingest"])
    graph = rng.choice(["rmat", "grid", "web"])
    if kind in ("ppr", "adjoint"):
        graph = rng.choice(["rmat", "web"])
    top = {"static": {"rmat": 1 << 22, "grid": 4096 ** 2, "web": 15_000_000},
           "dynamic": {"rmat": 1 << 20, "grid": 2000 ** 2, "web": 4_000_000},
           "update": {"rmat": 1 << 20, "grid": 2000 ** 2, "web": 3_000_000},
           "ppr": {"rmat": 1 << 19, "web": 300_000},
           "adjoint": {"rmat": 1 << 18, "web": 150_000},
           "ingest": {"rmat": 1 << 21, "grid": 3000 ** 2, "web": 3_000_000}}[kind][graph]
    n = _log(rng, 1000, top)
    if graph == "rmat":
        n = 1 << int(round(math.log2(n)))
    elif graph == "grid":
        n = int(math.isqrt(n)) ** 2
    else:
        n |= 1
    case = {"kind": kind, "graph": graph, "n": n, "salt": rng.randrange(1 << 20)}
    if kind == "static":
        case["refine"] = rng.random() < 0.3
    if kind == "dynamic":
        case["mode"] = rng.choice(["nd", "dt", "df", "dfp"])
    if kind in ("dynamic", "update"):
        case["batch"] = _log(rng, 2, max(4, n // 100))
    if kind == "ppr":
        case["vectors"] = rng.randint(1, 64)
        case["refine"] = rng.random() < 0.5
    return case


# ---- inputs ----------------------------------------------------------------------
def _gen(case, seed):
    g = torch.Generator(device=DEV)
    if case["kind"] == "adjoint":   # a training run keeps its graph: the seed draws weights, teleport and goal
        seed = 0
    g.manual_seed(seed * 1000003 + case.get("salt", 0) * 7919 + case["n"])
    return g


def _rmat(n, g):
    """16 draws a vertex, one quadrant of the adjacency matrix a level."""
    m = 16 * n
    u = torch.zeros(m, dtype=torch.int32, device=DEV)
    v = torch.zeros(m, dtype=torch.int32, device=DEV)
    for _ in range(n.bit_length() - 1):
        x = torch.rand(m, generator=g, device=DEV)
        u.mul_(2).add_((x >= 0.76).int())
        v.mul_(2).add_((((x >= 0.57) & (x < 0.76)) | (x >= 0.95)).int())
    return u, v


def _web(n, g):
    """Out-degrees floor(5.5 * U^(-1/1.1)) up to 100,000 (40 on average), 70%
    of the targets within 4096 ids of their source, the rest uniform."""
    x = torch.rand(n, generator=g, device=DEV, dtype=torch.float64).clamp_(min=1e-12)
    deg = (5.5 * x ** (-1 / 1.1)).clamp_(max=min(100_000, max(16, n // 4))).long()
    u = torch.repeat_interleave(torch.arange(n, dtype=torch.int32, device=DEV), deg)
    m = u.numel()
    window = min(4096, max(1, n // 8))
    v = torch.randint(-window, window + 1, (m,), generator=g, device=DEV, dtype=torch.int32)
    v.add_(u).remainder_(n)
    far = torch.rand(m, generator=g, device=DEV) >= 0.7
    v = torch.where(far, torch.randint(0, n, (m,), generator=g, device=DEV, dtype=torch.int32), v)
    return u, v


def _grid(n, g):
    """4 neighbours both ways and a diagonal pair from 5% of the vertices."""
    w = math.isqrt(n)
    at = torch.arange(n, dtype=torch.int32, device=DEV).view(w, w)
    right = (at[:, :-1].reshape(-1), at[:, 1:].reshape(-1))
    down = (at[:-1].reshape(-1), at[1:].reshape(-1))
    pick = torch.rand((w - 1, w - 1), generator=g, device=DEV) < 0.05
    diag = (at[:-1, :-1][pick], at[1:, 1:][pick])
    a = torch.cat([right[0], down[0], diag[0]])
    b = torch.cat([right[1], down[1], diag[1]])
    return torch.cat([a, b]), torch.cat([b, a])


def _edges(case, g):
    u, v = {"rmat": _rmat, "web": _web, "grid": _grid}[case["graph"]](case["n"], g)
    return u.contiguous(), v.contiguous()


def _batch(case, u, v, g):
    """A raw batch: half deletions of drawn edges, half insertions of uniform
    pairs (as (del_u, del_v, ins_u, ins_v) on the GPU)."""
    k = max(1, case["batch"] // 2)
    at = torch.randint(0, u.numel(), (k,), generator=g, device=DEV)
    du, dv = u[at], v[at]
    keep = du != dv
    iu = torch.randint(0, case["n"], (k,), generator=g, device=DEV, dtype=torch.int32)
    iv = torch.randint(0, case["n"], (k,), generator=g, device=DEV, dtype=torch.int32)
    return du[keep], dv[keep], iu, iv


def _host(t):
    return t.cpu().numpy().view(np.uint32)


def _device(a):
    return torch.from_numpy(a.view(np.int32)).to(DEV)


def _seeds(case, seed):
    """Teleport sets, sizes log-uniform in 1 .. 1000."""
    r = np.random.default_rng([seed, case["n"], case.get("salt", 0)])
    return [r.integers(0, case["n"], int(round(math.exp(r.uniform(0, math.log(1000)))))).astype(np.uint32)
            for _ in range(case["vectors"])]


def _options(case):
    return pg.options(precision=pg.FP32_REFINE if case.get("refine") else pg.FP64)


# ---- what a program has before the call ------------------------------------------
def prepare(case, seed):
    g = _gen(case, seed)
    u, v = _edges(case, g)
    n, kind = case["n"], case["kind"]
    s = {"case": case, "opts": _options(case)}
    if kind == "ingest":
        s.update(u=u, v=v)
        return s
    graph = pg.Graph.from_device_edges(ctx(), n, u, v)
    s["graph"] = graph
    if kind in ("dynamic", "update"):
        raw = [_host(x) for x in _batch(case, u, v, g)]
        s["q"] = torch.empty(n, dtype=torch.float64, device=DEV)
        pg.solve_device(ctx(), graph, pg.STATIC, None, s["q"].data_ptr())
        if kind == "update":
            s["raw"] = raw
        else:
            tidy = graph.tidy_batch(*raw)
            graph.apply_batch(*tidy)
            s["batch"] = [_device(x) for x in tidy]
    if kind == "ppr":
        s["seeds"] = _seeds(case, seed)
    if kind == "adjoint":
        g.manual_seed(seed)
        m = graph.size()[1]
        s["weights"] = (0.5 + 1.5 * torch.rand(m, generator=g, device=DEV)).requires_grad_(True)
        t = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
        s["teleport"] = (t / t.sum()).requires_grad_(True)
        s["alpha"] = torch.tensor(ALPHA, dtype=torch.float64, device=DEV, requires_grad=True)
        s["goal"] = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    del u, v
    return s


# ---- one pass --------------------------------------------------------------------
def _solve_dynamic(s, mode, batch):
    ranks = torch.empty_like(s["q"])
    du, dv, iu, iv = batch
    ptrs = (du.data_ptr() or None, dv.data_ptr() or None, du.numel(),
            iu.data_ptr() or None, iv.data_ptr() or None, iu.numel())
    res = pg.solve_device(ctx(), s["graph"], getattr(pg, MODES[mode]), s["q"].data_ptr(), ranks.data_ptr(), ptrs,
                          s["opts"])
    return {"ranks": ranks, "iterations": res["iterations"]}


def run(s):
    case = s["case"]
    kind, n = case["kind"], case["n"]
    if kind == "static" and n <= 4096:   # a small result comes back to the host
        ranks, res = pg.pagerank_static(ctx(), s["graph"], s["opts"])
        return {"ranks": ranks} if case["refine"] else {"ranks": ranks, "iterations": res["iterations"]}
    if kind in ("static", "ingest"):
        graph = s["graph"] if kind == "static" else pg.Graph.from_device_edges(ctx(), n, s["u"], s["v"])
        ranks = torch.empty(n, dtype=torch.float64, device=DEV)
        res = pg.solve_device(ctx(), graph, pg.STATIC, None, ranks.data_ptr(), opts=s["opts"])
        return {"ranks": ranks} if case.get("refine") else {"ranks": ranks, "iterations": res["iterations"]}
    if kind == "dynamic":
        return _solve_dynamic(s, case["mode"], s["batch"])
    if kind == "update":
        graph = s["graph"]
        tidy = graph.tidy_batch(*s["raw"])
        graph.apply_batch(*tidy)
        batch = [_device(x) for x in tidy]
        torch.cuda.current_stream().synchronize()   # the library works on its own stream
        out = _solve_dynamic(s, "dfp", batch)
        graph.apply_batch(tidy[2], tidy[3], tidy[0], tidy[1])
        return out
    if kind == "ppr":
        ranks = torch.empty((n, case["vectors"]), dtype=torch.float64, device=DEV)
        pg.solve_ppr_batched_device(ctx(), s["graph"], s["seeds"], ranks.data_ptr(), s["opts"])
        return {"ranks": ranks}
    from pagerank_gb300.autograd import weighted_pagerank
    r = weighted_pagerank(ctx(), s["graph"], s["weights"], s["teleport"], s["alpha"])
    loss = (s["goal"] * r).sum()
    gw, gt, ga = torch.autograd.grad(loss, (s["weights"], s["teleport"], s["alpha"]))
    return {"ranks": r.detach(), "grad_weights": gw, "grad_teleport": gt, "grad_alpha": ga}


# ---- the least a pass has to move --------------------------------------------------
# edges a vertex, and sweeps from uniform ranks to 1e-10 (personalized ones: from the teleport rows)
SHAPE = {"rmat": {"deg": 16.0, "sweeps": 70, "ppr": 70}, "web": {"deg": 36.0, "sweeps": 8, "ppr": 27},
         "grid": {"deg": 5.1, "sweeps": 10}}


def work(case):
    n, kind = case["n"], case["kind"]
    m = n * SHAPE[case["graph"]]["deg"]
    sweeps = SHAPE[case["graph"]]["sweeps"]
    if kind == "static":     # 4 bytes an edge, 8 a gathered value, 20 a vertex, a sweep (half the values in FP32)
        per = 8 * m + 12 * n if case["refine"] else 12 * m + 20 * n
        return {"bytes": sweeps * per, "flops": sweeps * m}
    if kind == "dynamic":    # one sweep over the graph, its previous and its new ranks
        return {"bytes": 12 * m + 36 * n, "flops": m}
    if kind == "update":     # both CSRs read and written twice (the batch and its rollback), one sweep
        return {"bytes": 2 * 16 * m + 12 * m + 36 * n, "flops": m}
    if kind == "ppr":        # one row of the vectors' values an edge and three a vertex, a sweep
        size = 4 if case["refine"] else 8
        cols, sweeps = case["vectors"], SHAPE[case["graph"]]["ppr"]
        return {"bytes": sweeps * ((4 + size * cols) * m + 3 * size * cols * n), "flops": 2 * sweeps * m * cols}
    if kind == "adjoint":    # 4 + 8 + 8 bytes an edge a sweep, both ways to 1e-12, and the weights and gradients
        return {"bytes": 270 * (20 * m + 24 * n) + 40 * m, "flops": 270 * 2 * m}
    return {"bytes": 16 * n * 8 + 8 * m + sweeps * (12 * m + 20 * n), "flops": sweeps * m}


# ---- the same in 64 bits by torch alone --------------------------------------------
def _keys(u, v, n):
    loops = torch.arange(n, device=DEV)
    return torch.unique(torch.cat([u.long() * n + v, loops * n + loops]))


def _parts(key, n):
    u, v = key // n, key % n
    return u, v, torch.bincount(u, minlength=n).double()


def _pull(u, v, x):
    """sum of x[u] over the edges u -> v, per v."""
    out = torch.zeros_like(x)
    step = max(1, (1 << 28) // max(1, x[:1].numel()))
    for i in range(0, u.numel(), step):
        out.index_add_(0, v[i:i + step], x[u[i:i + step]])
    return out


def _jacobi(u, v, d, r, base, tol, cap=2000):
    for _ in range(cap):
        a = base + ALPHA * _pull(u, v, r / d)
        delta = (a - r).abs().max().item()
        r = a
        if delta < tol:
            break
    return r


def _static(u, v, d, n, tol):
    return _jacobi(u, v, d, torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV), (1 - ALPHA) / n, tol)


def _out_mark(u, v, src, flags):
    flags[v[src[u]]] = True
    return flags


def _dynamic(case, key, raw, n, mode):
    """The library's dynamic modes as mask operations on whole arrays."""
    u, v, d = _parts(key, n)
    q = _static(u, v, d, n, TOL)
    du, dv, iu, iv = (x.long() for x in raw)
    dele = torch.unique(du * n + dv)
    ins = torch.unique(iu * n + iv)
    ins = ins[~torch.isin(ins, key)]
    key = torch.cat([key[~torch.isin(key, dele)], ins])
    u, v, d = _parts(key, n)
    if mode == "nd":
        return _jacobi(u, v, d, q, (1 - ALPHA) / n, TOL, CAP)
    src = torch.zeros(n, dtype=torch.bool, device=DEV)
    src[dele // n] = True
    src[ins // n] = True
    hit = torch.zeros(n, dtype=torch.bool, device=DEV)
    hit[dele % n] = True
    if dele.numel() + ins.numel():
        _out_mark(u, v, src, hit)
    if mode == "dt":
        size = -1
        while size != int(hit.sum()):
            size = int(hit.sum())
            for _ in range(16):
                _out_mark(u, v, hit.clone(), hit)
    r = q
    for _ in range(CAP):
        c = _pull(u, v, r / d)
        if mode == "dfp":
            a = ((1 - ALPHA) / n + ALPHA * (c - r / d)) * (1 / (1 - ALPHA / d))
        else:
            a = (1 - ALPHA) / n + ALPHA * c
        a = torch.where(hit, a, r)
        delta = (a - r).abs()
        rel = delta / torch.maximum(a, r)
        moved = hit & (rel > 1e-6)
        if mode == "dfp":
            hit = hit & ~(rel <= 1e-6)
        if mode != "dt":
            hit = _out_mark(u, v, moved, hit.clone())
        r = a
        if delta.max().item() < TOL:
            break
    return r


def exact(case, seed):
    g = _gen(case, seed)
    u, v = _edges(case, g)
    n, kind = case["n"], case["kind"]
    key = _keys(u, v, n)
    if kind in ("dynamic", "update"):
        mode = case.get("mode", "dfp")
        raw = _batch(case, u, v, g)
        return {"ranks": _dynamic(case, key, raw, n, mode), "iterations": None}
    u, v, d = _parts(key, n)
    if kind in ("static", "ingest"):
        # the refinement's answer is the converged ranks, the drop-in's the iterate that passes the test
        if case.get("refine"):
            return {"ranks": _static(u, v, d, n, 1e-17)}
        r = _static(u, v, d, n, TOL)
        return {"ranks": r if n > 4096 or kind == "ingest" else r.cpu().numpy(), "iterations": None}
    if kind == "ppr":
        t = torch.zeros((n, case["vectors"]), dtype=torch.float64, device=DEV)
        for k, x in enumerate(_seeds(case, seed)):
            at = torch.from_numpy(x.astype(np.int64)).to(DEV)
            t[:, k].index_add_(0, at, torch.full((len(x),), 1.0 / len(x), dtype=torch.float64, device=DEV))
        back = torch.argsort(v, stable=True)
        off = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
        off[1:] = torch.cumsum(torch.bincount(v, minlength=n), 0)
        A = torch.sparse_csr_tensor(off, u[back], torch.ones(u.numel(), dtype=torch.float64, device=DEV), (n, n))
        r = t.clone()
        for _ in range(2000):
            a = (1 - ALPHA) * t + ALPHA * (A @ (r / d[:, None]))
            delta = (a - r).abs().max().item()
            r = a
            if delta < (1e-16 if case["refine"] else TOL):
                break
        return {"ranks": r}
    g.manual_seed(seed)
    m = u.numel()
    w = (0.5 + 1.5 * torch.rand(m, generator=g, device=DEV)).double()
    t = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    t = t / t.sum()
    goal = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    W = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, u, w)
    p = w / W[u]
    r, lam = t, goal
    for _ in range(400):
        r = (1 - ALPHA) * t + ALPHA * torch.zeros_like(r).index_add_(0, v, p * r[u])
        lam = goal + ALPHA * torch.zeros_like(r).index_add_(0, u, p * lam[v])
    y = torch.zeros_like(r).index_add_(0, v, p * r[u])
    gw = r[u] / W[u] * (ALPHA * lam[v] - lam[u] + goal[u])
    return {"ranks": r, "grad_weights": gw, "grad_teleport": (1 - ALPHA) * lam, "grad_alpha": (lam * (y - t)).sum()}
