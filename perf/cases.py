"""The work that programs built on this library have it do, as timed cases.

Every case is one call (or one call chain) of the Python entry points in
apspie_b200.ops on device-resident inputs that are built here with torch from
a seed: R-MAT graphs (0.57, 0.19, 0.19, 0.05), Erdos-Renyi graphs, 5-point
grids and matrices with power-law rows, in the sizes of this repository's
benchmark, tests and workloads.  The edges of a random graph are drawn once
per size and the seed numbers the vertices, so that outputs whose length
depends on the structure have one length for all seeds.  listed() names twelve of them, draw() gives
others of the same ranges: from a thousand vertices, where launches and
latency count, to the benchmark's full sizes, odd sizes among them.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

import apspie_b200 as ap
from apspie_b200.graph import DeviceGraph

SEMIRINGS = {"plus_times": 0, "min_plus": 1, "max_times": 2, "or_and": 3}


def listed() -> list[dict]:
    return [
        # BFS query on a small graph: a program that asks for many short
        # traversals; launch and barrier latency is all there is
        {"name": "bfs_rmat14", "op": "bfs", "graph": "rmat", "scale": 14, "ef": 16, "sym": True},
        # the benchmark's headline: BFS of a large social-network-like graph,
        # few levels, direction-switching
        {"name": "bfs_rmat22", "op": "bfs", "graph": "rmat", "scale": 22, "ef": 16, "sym": True},
        # BFS of a mesh / road-like graph: about a thousand thin levels
        {"name": "bfs_grid1024", "op": "bfs", "graph": "grid", "rows": 1024, "cols": 1024},
        # shortest paths on a directed scale-free graph, both weight types
        {"name": "sssp_u32_rmat20", "op": "sssp", "graph": "rmat", "scale": 20, "ef": 16,
         "sym": False, "weights": "u32"},
        {"name": "sssp_f32_rmat20", "op": "sssp", "graph": "rmat", "scale": 20, "ef": 16,
         "sym": False, "weights": "f32"},
        # maximal independent set (colouring / coarsening step) of a sparse
        # random graph
        {"name": "mis_er20", "op": "mis", "graph": "er", "n": 1 << 20, "deg": 8, "delta": 1.0},
        # triangle count of a scale-free graph, from the graph to the count:
        # degree relabel, lower triangle, masked product
        {"name": "tc_rmat18", "op": "tc", "graph": "rmat", "scale": 18, "ef": 16, "sym": True},
        # sparse matrix product of the benchmark: 2^18 power-law rows
        {"name": "spgemm_powerlaw18", "op": "spgemm", "m": 1 << 18, "k": 1 << 18, "n": 1 << 18,
         "mean": 16, "max_deg": 4096},
        # dense SpMV (one PageRank-like step) on a scale-free matrix
        {"name": "spmv_rmat20", "op": "spmv", "graph": "rmat", "scale": 20, "ef": 16, "sym": True,
         "semiring": "plus_times", "val": True},
        # sparse vector times matrix, every 64th vertex in the frontier
        {"name": "spmspv_rmat20", "op": "spmspv", "graph": "rmat", "scale": 20, "ef": 16,
         "sym": True, "semiring": "plus_times", "val": True, "every": 64},
        # transpose with values: the in-adjacency of a directed weighted graph
        {"name": "transpose_rmat20", "op": "transpose", "graph": "rmat", "scale": 20, "ef": 16,
         "sym": False},
        # many traversals of uneven graphs in one call, a deep grid among them
        {"name": "batch_uneven", "op": "batch", "scales": "12,16,18", "grid": 128, "bfs": 48,
         "sssp": 12},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, max_scale: int, max_er: int, max_side: int, sym=None) -> dict:
    """max_side 0: no grids."""
    kind = rng.choice(["rmat", "rmat", "er", "grid"] if max_side else ["rmat", "rmat", "er"])
    if kind == "rmat":
        return {"graph": "rmat", "scale": rng.randint(10, max_scale), "ef": rng.randint(5, 16),
                "sym": rng.random() < 0.6 if sym is None else sym}
    if kind == "er":
        return {"graph": "er", "n": _log_int(rng, 1000, max_er), "deg": rng.randint(3, 16)}
    return {"graph": "grid", "rows": _log_int(rng, 24, max_side), "cols": _log_int(rng, 24, max_side)}


def draw(rng) -> dict:
    op = rng.choice(["bfs", "bfs", "sssp", "sssp", "mis", "tc", "spgemm", "spgemm", "spmv",
                     "spmspv", "transpose", "batch"])
    if op == "bfs":
        return {"op": op, **_draw_graph(rng, 21, 1 << 21, 700)}
    if op == "sssp":
        return {"op": op, **_draw_graph(rng, 20, 1 << 19, 300),
                "weights": rng.choice(["u32", "f32"])}
    if op == "mis":
        return {"op": op, **_draw_graph(rng, 20, 1 << 20, 1024, sym=True),
                "delta": rng.choice([1.0, 1.0, 0.1])}
    if op == "tc":
        return {"op": op, **_draw_graph(rng, 17, 1 << 20, 0, sym=True)}
    if op == "spgemm":
        m = _log_int(rng, 1000, 200000)
        square = rng.random() < 0.5
        k, n = (m, m) if square else (_log_int(rng, 1000, 200000), _log_int(rng, 1000, 400000))
        return {"op": op, "m": m, "k": k, "n": n, "mean": rng.randint(4, 14),
                "max_deg": _log_int(rng, 64, 2000)}
    if op == "spmv":
        return {"op": op, **_draw_graph(rng, 20, 1 << 20, 1024),
                "semiring": rng.choice(["plus_times", "plus_times", "min_plus", "max_times",
                                        "or_and"]), "val": rng.random() < 0.8}
    if op == "spmspv":
        return {"op": op, **_draw_graph(rng, 20, 1 << 20, 0),
                "semiring": rng.choice(["plus_times", "plus_times", "min_plus", "max_times",
                                        "or_and"]), "val": rng.random() < 0.8,
                "every": _log_int(rng, 2, 500)}
    if op == "transpose":
        return {"op": op, **_draw_graph(rng, 20, 1 << 20, 1024)}
    scales = sorted(rng.sample([10, 11, 12, 13, 14, 15, 16, 17], rng.randint(1, 3)))
    return {"op": op, "scales": ",".join(str(s) for s in scales),
            "grid": rng.choice([0, 0, _log_int(rng, 24, 100)]), "bfs": rng.randint(3, 64),
            "sssp": rng.randint(1, 16)}


# ------------------------------------------------------------------ inputs --

def _device() -> torch.device:
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _csr(keys: torch.Tensor, m: int, n: int):
    """CSR of the distinct row * n + col keys, columns ascending in a row."""
    keys = torch.unique(keys)
    rows = keys // n
    ptr = torch.zeros(m + 1, dtype=torch.int64, device=keys.device)
    ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    return ptr.to(torch.int32), (keys - rows * n).to(torch.int32)


def _renumber(m: int, gen: torch.Generator) -> torch.Tensor:
    return torch.randperm(m, generator=gen, device=gen.device)


def _rmat(scale: int, ef: int, sym: bool, perm: torch.Tensor):
    m = 1 << scale
    gen = _generator(1)
    dev = gen.device
    r = torch.zeros(ef * m, dtype=torch.int64, device=dev)
    c = torch.zeros_like(r)
    for _ in range(scale):
        u = torch.rand(ef * m, generator=gen, device=dev)
        low = u >= 0.76  # (0.57, 0.19 | 0.19, 0.05)
        right = (u >= 0.95) | ((u >= 0.57) & ~low)
        r = (r << 1) | low
        c = (c << 1) | right
    r, c = perm[r], perm[c]
    keep = r != c
    r, c = r[keep], c[keep]
    keys = r * m + c
    return m, *_csr(torch.cat([keys, c * m + r]) if sym else keys, m, m)


def _er(n: int, deg: int, perm: torch.Tensor):
    gen = _generator(2)
    e = torch.randint(0, n, (2, n * deg // 2), generator=gen, device=gen.device)
    r, c = perm[e[0]], perm[e[1]]
    keep = r != c
    r, c = r[keep], c[keep]
    return n, *_csr(torch.cat([r * n + c, c * n + r]), n, n)


def _grid(rows: int, cols: int):
    """5-point grid, neighbours ascending: up, left, right, down."""
    m = rows * cols
    v = torch.arange(m, device=_device())
    y, x = v // cols, v % cols
    keys = [v * m + v + d for d in (-cols, -1, 1, cols)]
    ok = [y > 0, x > 0, x < cols - 1, y < rows - 1]
    return m, *_csr(torch.cat([k[o] for k, o in zip(keys, ok)]), m, m)


def _graph(case: dict, gen: torch.Generator):
    """(m, ptr, ind, symmetric) of a case's graph and its vertices' numbers."""
    if case["graph"] == "grid":
        return *_grid(case["rows"], case["cols"]), True, None
    perm = _renumber(1 << case["scale"] if case["graph"] == "rmat" else case["n"], gen)
    if case["graph"] == "rmat":
        return *_rmat(case["scale"], case["ef"], case["sym"], perm), case["sym"], perm
    return *_er(case["n"], case["deg"], perm), True, perm


def _sources(ptr: torch.Tensor, count: int, gen: torch.Generator) -> list[int]:
    """Random vertices among those of at least average degree: they lie in
    the giant component."""
    deg = ptr[1:] - ptr[:-1]
    ok = torch.nonzero(deg >= torch.clamp(deg.double().mean().floor(), min=1.0)).flatten()
    return ok[torch.randint(0, len(ok), (count,), generator=gen, device=gen.device)].tolist()


def _uniform(n: int, lo: float, hi: float, gen: torch.Generator) -> torch.Tensor:
    return torch.rand(n, generator=gen, device=gen.device) * (hi - lo) + lo


def _weights_f32(n: int, gen: torch.Generator) -> torch.Tensor:
    return 1.0 - torch.rand(n, generator=gen, device=gen.device)  # (0, 1]


def _powerlaw_xmin(mean: float, top: float, alpha: float = 2.1) -> float:
    """x_min of a Pareto(alpha) truncated at `top` whose floor has this mean."""
    u = (np.arange(20000) + 0.5) / 20000
    lo, hi = 0.1, float(mean) + 1.0
    for _ in range(30):
        x = 0.5 * (lo + hi)
        got = np.floor(x * (1 - u * (1 - (x / top) ** (alpha - 1))) ** (-1 / (alpha - 1))).mean()
        lo, hi = (x, hi) if got < mean else (lo, x)
    return 0.5 * (lo + hi)


def _powerlaw(rowno: torch.Tensor, colno: torch.Tensor, mean: float, max_deg: int,
              gen: torch.Generator, alpha: float = 2.1):
    """Matrix with power-law row lengths, uniform columns and values in
    [-1, 1]; rowno and colno number its rows and columns."""
    m, n = len(rowno), len(colno)
    base = _generator(3)
    top = float(min(max_deg, n // 2) + 1)
    xmin = _powerlaw_xmin(mean, top, alpha)
    u = torch.rand(m, generator=base, device=base.device, dtype=torch.float64)
    tail = (xmin / top) ** (alpha - 1)
    deg = torch.floor(xmin * (1 - u * (1 - tail)) ** (-1 / (alpha - 1))).to(torch.int64)
    rows = torch.repeat_interleave(torch.arange(m, device=gen.device), deg)
    cols = torch.randint(0, n, (len(rows),), generator=base, device=base.device)
    ptr, ind = _csr(rowno[rows] * n + colno[cols], m, n)
    return ptr, ind, _uniform(len(ind), -1.0, 1.0, gen)


def _inputs(case: dict, seed: int) -> SimpleNamespace:
    """The case's inputs, without this library: used by prepare and exact."""
    gen = _generator(seed)
    op = case["op"]
    s = SimpleNamespace(op=op)
    if op == "spgemm":
        m, k, n = case["m"], case["k"], case["n"]
        square = m == k == n
        mid = _renumber(k, gen)
        s.A = (m, k, *_powerlaw(mid if square else _renumber(m, gen), mid, case["mean"],
                                case["max_deg"], gen))
        s.B = s.A if square else (k, n, *_powerlaw(mid, _renumber(n, gen), case["mean"],
                                                   case["max_deg"], gen))
        return s
    if op == "batch":
        s.graphs = [_rmat(int(sc), 16, True, _renumber(1 << int(sc), gen))
                    for sc in case["scales"].split(",")]
        if case["grid"]:
            s.graphs.append(_grid(case["grid"], case["grid"]))
        s.weights = [torch.randint(1, 256, (len(ind),), generator=gen, device=gen.device,
                                   dtype=torch.int32) for _, _, ind in s.graphs]
        s.sources = [_sources(ptr, case["bfs"] + case["sssp"], gen) for _, ptr, _ in s.graphs]
        return s
    s.m, s.ptr, s.ind, s.sym, perm = _graph(case, gen)
    nnz = len(s.ind)
    if op in ("bfs", "sssp"):
        s.src = _sources(s.ptr, 1, gen)[0]
    if op == "sssp":
        s.w_u32 = s.w_f32 = None
        if case["weights"] == "u32":
            s.w_u32 = torch.randint(1, 256, (nnz,), generator=gen, device=gen.device,
                                    dtype=torch.int32)
        else:
            s.w_f32 = _weights_f32(nnz, gen)
    if op in ("spmv", "spmspv", "transpose"):
        s.val = _weights_f32(nnz, gen) if case.get("val", True) else None
    if op == "spmv":
        s.x = torch.rand(s.m, generator=gen, device=gen.device)
        s.sr = SEMIRINGS[case["semiring"]]
    if op == "spmspv":
        s.xind = torch.sort(perm[::case["every"]])[0].to(torch.int32)
        s.xval = torch.rand(len(s.xind), generator=gen, device=gen.device)
        s.sr = SEMIRINGS[case["semiring"]]
    return s


def prepare(case: dict, seed: int) -> SimpleNamespace:
    s = _inputs(case, seed)
    s.ctx = ap.Context(0)
    if s.op == "batch":
        s.jobs = []
        for (m, ptr, ind), w, src in zip(s.graphs, s.weights, s.sources):
            g = DeviceGraph(m, len(ind), ptr, ind, w_u32=w, symmetric=True)
            s.jobs.append({"type": "bfs", "graph": g, "sources": src[:case["bfs"]]})
            s.jobs.append({"type": "sssp", "graph": g, "sources": src[case["bfs"]:]})
    elif s.op != "spgemm":
        s.g = DeviceGraph(s.m, len(s.ind), s.ptr, s.ind, w_u32=getattr(s, "w_u32", None),
                          w_f32=getattr(s, "w_f32", None), symmetric=s.sym)
    if s.op == "sssp":
        s.weights = case["weights"]
    if s.op == "mis":
        s.delta = case["delta"]
        s.prio = torch.from_numpy(ap.mt19937(seed % (1 << 32), s.m).view(np.int32)).to(_device())
    return s


def run(s: SimpleNamespace):
    if s.op == "bfs":
        return ap.bfs(s.ctx, s.g, s.src)
    if s.op == "sssp":
        return ap.sssp(s.ctx, s.g, s.src, weights=s.weights)
    if s.op == "mis":
        return ap.mis(s.ctx, s.g, s.prio, delta=s.delta)
    if s.op == "tc":
        perm, lptr, lind = ap.tc_prepare(s.ctx, s.g)
        return [perm, lptr, lind, ap.triangle_count(s.ctx, s.m, lptr, lind)]
    if s.op == "spgemm":
        return list(ap.spgemm(s.ctx, s.A, s.B))
    if s.op == "spmv":
        return ap.spmv(s.ctx, s.m, s.ptr, s.ind, s.val, s.x, s.sr)
    if s.op == "spmspv":
        return list(ap.spmspv(s.ctx, s.sr, s.g, s.xind, s.xval, s.val))
    if s.op == "transpose":
        return list(ap.csr_transpose(s.ctx, s.m, s.m, s.ptr, s.ind, s.val))
    return ap.batch_run(s.ctx, s.jobs)


# -------------------------------------------------------------------- work --

def _graph_size(case: dict) -> tuple[int, int]:
    """(m, about nnz): repeated samples of an R-MAT graph, some 7 %, are dropped."""
    if case["graph"] == "rmat":
        m = 1 << case["scale"]
        return m, int(0.93 * case["ef"] * m * (2 if case["sym"] else 1))
    if case["graph"] == "er":
        return case["n"], case["n"] * case["deg"]
    return case["rows"] * case["cols"], 4 * case["rows"] * case["cols"]


def work(case: dict) -> dict:
    op = case["op"]
    if op == "spgemm":
        # A and B read once, C (about one entry per product) written once
        prods = case["m"] * case["mean"] * case["mean"]
        bytes_ = 8 * (case["m"] + case["k"]) * case["mean"] + 8 * prods + 4 * case["m"]
        return {"bytes": bytes_, "flops": 2 * prods}
    if op == "batch":
        bytes_ = 0
        sizes = [_graph_size({"graph": "rmat", "scale": int(sc), "ef": 16, "sym": True})
                 for sc in case["scales"].split(",")]
        if case["grid"]:
            sizes.append((case["grid"] ** 2, 4 * case["grid"] ** 2))
        for m, nnz in sizes:  # the graph and its weights once, every answer once
            bytes_ += 8 * nnz + 4 * m + 4 * m * (case["bfs"] + case["sssp"])
        return {"bytes": bytes_, "flops": 0}
    m, nnz = _graph_size(case)
    if op == "bfs":  # indices and offsets of the reached vertices, the depths
        return {"bytes": 4 * nnz + 4 * m + 4 * m, "flops": 0}
    if op == "sssp":
        return {"bytes": 8 * nnz + 4 * m + 4 * m, "flops": nnz}
    if op == "mis":  # indices, offsets, priorities, membership
        return {"bytes": 4 * nnz + 12 * m, "flops": 0}
    if op == "tc":  # the graph, the permutation, L
        return {"bytes": 4 * nnz + 4 * m + 4 * m + 4 * m + 2 * nnz, "flops": 0}
    if op == "spmv":
        return {"bytes": 4 * m + (8 if case["val"] else 4) * nnz + 8 * m, "flops": 2 * nnz}
    if op == "spmspv":
        share = 1.0 / case["every"]
        e = nnz * share
        return {"bytes": int((8 if case["val"] else 4) * e + 16 * m * share + 8 * min(m, e)),
                "flops": 2 * int(e)}
    return {"bytes": 16 * nnz + 8 * m, "flops": 0}  # transpose: read and written once


# ------------------------------------------------------------------- exact --

def _exact_reduce(sr: int, rows: torch.Tensor, terms: torch.Tensor, n: int) -> torch.Tensor:
    if sr == 0:
        return torch.zeros(n, dtype=torch.float64, device=rows.device).index_add_(0, rows, terms)
    big = float(np.finfo(np.float32).max)
    start = {1: big, 2: -big, 3: 0.0}[sr]
    out = torch.full((n,), start, dtype=torch.float64, device=rows.device)
    return out.scatter_reduce_(0, rows, terms, "amin" if sr == 1 else "amax")


def _exact_terms(sr: int, a: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    if sr == 1:
        return a + x
    if sr == 3:
        return ((a != 0) & (x != 0)).double()
    return a * x


def _row_ids(ptr: torch.Tensor) -> torch.Tensor:
    return torch.repeat_interleave(torch.arange(len(ptr) - 1, device=ptr.device),
                                   (ptr[1:] - ptr[:-1]).long())


def _expand(ptr: torch.Tensor, rows: torch.Tensor):
    """(owner position, entry position) of every entry of the listed rows."""
    start = ptr[rows].long()
    deg = ptr[rows + 1].long() - start
    owner = torch.repeat_interleave(torch.arange(len(rows), device=ptr.device), deg)
    first = torch.cumsum(deg, 0) - deg
    return owner, torch.arange(len(owner), device=ptr.device) - first[owner] + start[owner]


def exact(case: dict, seed: int):
    op = case["op"]
    if op == "sssp" and case["weights"] == "f32":
        s = _inputs(case, seed)
        src, dst, w = _row_ids(s.ptr), s.ind.long(), s.w_f32.double()
        dist = torch.full((s.m,), math.inf, dtype=torch.float64, device=w.device)
        dist[s.src] = 0.0
        while True:  # Bellman-Ford to its fixed point
            new = dist.scatter_reduce(0, dst, dist[src] + w, "amin")
            if torch.equal(new, dist):
                return dist
            dist = new
    if op == "spmv":
        s = _inputs(case, seed)
        a = torch.ones(len(s.ind), dtype=torch.float64, device=s.ptr.device) if s.val is None \
            else s.val.double()
        terms = _exact_terms(s.sr, a, s.x.double()[s.ind.long()])
        return _exact_reduce(s.sr, _row_ids(s.ptr), terms, s.m)
    if op == "spmspv":
        s = _inputs(case, seed)
        owner, pos = _expand(s.ptr, s.xind.long())
        a = torch.ones(len(pos), dtype=torch.float64, device=pos.device) if s.val is None \
            else s.val.double()[pos]
        rows = s.ind.long()[pos]
        terms = torch.ones_like(a) if s.sr == 3 else \
            _exact_terms(s.sr, a, s.xval.double()[owner])
        y = _exact_reduce(s.sr, rows, terms, s.m)
        return [None, y[torch.unique(rows)], None]
    if op == "spgemm":
        s = _inputs(case, seed)
        (m, _, ap_, ai, av), (_, n, bp, bi, bv) = s.A, s.B
        owner, pos = _expand(bp, ai.long())
        keys = _row_ids(ap_)[owner] * n + bi.long()[pos]
        terms = av.double()[owner] * bv.double()[pos]
        del owner, pos
        _, at = torch.unique(keys, return_inverse=True)
        return [None, None, torch.zeros(int(at.max()) + 1, dtype=torch.float64,
                                        device=at.device).index_add_(0, at, terms)]
    if op == "transpose":  # values only move
        s = _inputs(case, seed)
        return [None, None, s.val.double()[torch.argsort(s.ind.long(), stable=True)]]
    return None  # whole numbers
