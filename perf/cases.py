"""Performance cases of the graph framework: one pass each through its public entry points.

Every case is a call that a program makes on a graph it keeps on the GPU: a traversal (one
source, up to 64 sources, one source per graph of a batch), shortest paths, connected
components, PageRank, or differentiable personalised PageRank with its backward pass. The
inputs are the synthetic families the framework is used on: power-law R-MAT graphs (A/B/C/D
.57/.19/.19/.05, vertices shuffled, duplicates and self-loops removed) and a road-like grid
with dropped edges and long shortcuts. They are drawn on the GPU from the seed, so another
seed is another graph, other weights and other sources.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import gpugraph_b200 as gg
from gpugraph_b200.ppr import ppr

UNREACHED_SSSP = int(gg.SSSP_INF)


# ---------------------------------------------------------------- the cases --
def _case(name, op, graph, size, ef=16, nsrc=1, nvec=0, wmax=0, extra=0):
    """op: the call. graph/size: "rmat" and "rmat_dir" of scale `size`, "road" of width `size`,
    "batch" of `size` R-MAT graphs. ef: edges per vertex drawn for an R-MAT graph. extra:
    isolated vertices appended (vertex counts that are no multiple of four). wmax: integer edge
    weights in [1, wmax]."""
    c = dict(op=op, graph=graph, size=size, ef=ef, nsrc=nsrc, nvec=nvec, wmax=wmax, extra=extra)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # A small graph explored interactively: the plain Python call, its depths back in host
        # memory and its statistics counted. Launches and latency, not bandwidth.
        _case("bfs_rmat16_host", "bfs_host", "rmat", 16),
        # One traversal of a graph of ordinary size, the depths staying on the GPU.
        _case("bfs_rmat21", "bfs", "rmat", 21, extra=1),
        # One traversal of a road network: many levels of small frontiers.
        _case("bfs_road1200", "bfs", "road", 1200),
        # 64 sources in one pass over a large power-law graph (centralities, landmark tables).
        _case("bfs_multi64_rmat22", "bfs_multi", "rmat", 22, nsrc=64),
        # Many small graphs of uneven size, one traversal each in the same launches.
        _case("bfs_batch256", "bfs_batch", "batch", 256, ef=8),
        # Shortest paths from one vertex, weights in [1, 64].
        _case("sssp_rmat21", "sssp", "rmat", 21, wmax=64),
        # Distance tables: an odd number of sources on a power-law graph, 64 on a road network.
        _case("sssp_multi37_rmat20", "sssp_multi", "rmat", 20, nsrc=37, wmax=64, extra=3),
        _case("sssp_multi64_road1200", "sssp_multi", "road", 1200, nsrc=64, wmax=1000),
        # Components of a power-law graph.
        _case("cc_rmat21", "cc", "rmat", 21),
        # Ranks of a directed power-law graph with dangling vertices, and of a road network.
        _case("pagerank_rmat22", "pagerank", "rmat_dir", 22),
        _case("pagerank_road1200", "pagerank", "road", 1200),
        # A training step through personalised PageRank: forward, and both gradients.
        _case("ppr_rmat20_32", "ppr", "rmat_dir", 20, nvec=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["bfs_host", "bfs", "bfs_pred", "bfs_roots", "bfs_multi", "bfs_batch", "sssp", "sssp_multi", "cc",
                     "pagerank", "ppr"])
    road = rng.random() < 0.35
    ef = rng.choice([4, 8, 12, 16])
    extra = rng.randrange(4)
    width = _log_int(rng, 64, 1200)
    if op == "bfs_batch":
        return _case("", op, "batch", _log_int(rng, 2, 256), ef=8)
    if op in ("bfs_host", "bfs", "bfs_pred", "bfs_roots", "sssp", "cc"):
        nsrc = rng.randint(2, 300) if op == "bfs_roots" else 1
        wmax = rng.choice([1, 64, 1000]) if op == "sssp" else 0
        if road:
            return _case("", op, "road", width, nsrc=nsrc, wmax=wmax)
        return _case("", op, "rmat", rng.randint(10, 21), ef=ef, nsrc=nsrc, wmax=wmax, extra=extra)
    if op in ("bfs_multi", "sssp_multi"):
        nsrc = rng.choice([64, rng.randint(1, 64)])
        wmax = rng.choice([1, 64, 1000]) if op == "sssp_multi" else 0
        if road:
            return _case("", op, "road", width, nsrc=nsrc, wmax=wmax)
        return _case("", op, "rmat", rng.randint(10, 20), ef=ef, nsrc=nsrc, wmax=wmax, extra=extra)
    if op == "pagerank":
        if road:
            return _case("", op, "road", width)
        return _case("", op, rng.choice(["rmat", "rmat_dir"]), rng.randint(10, 21), ef=ef, extra=extra)
    return _case("", op, "rmat_dir", rng.randint(9, 19), ef=ef, nvec=rng.choice([32, rng.randint(1, 64)]), extra=extra)


# --------------------------------------------------------------- the graphs --
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _rmat_edges(scales, ef, gen):
    """Edges of one R-MAT graph per entry of `scales`, with global vertex ids, and the graphs' first vertices."""
    sc = torch.tensor(scales, dtype=torch.int64, device="cuda")
    first = torch.zeros(len(scales) + 1, dtype=torch.int64, device="cuda")
    first[1:] = torch.cumsum(torch.ones_like(sc) << sc, 0)
    count = ef * (torch.ones_like(sc) << sc)
    m = int(count.sum())
    src = torch.zeros(m, dtype=torch.int64, device="cuda")
    dst = torch.zeros(m, dtype=torch.int64, device="cuda")
    bits = sc.repeat_interleave(count) if len(scales) > 1 else None
    for b in range(max(scales)):
        r = torch.rand(m, device="cuda", generator=gen)
        hi, lo = r >= 0.76, ((r >= 0.57) & (r < 0.76)) | (r >= 0.95)
        if bits is not None:
            hi, lo = hi & (b < bits), lo & (b < bits)
        src |= hi.to(torch.int64) << b
        dst |= lo.to(torch.int64) << b
    n = int(first[-1])
    if len(scales) > 1:
        base = first[:-1].repeat_interleave(count)
        src += base
        dst += base
        # shuffled within each graph: vertices sorted by (graph, random key)
        graph = torch.arange(len(scales), device="cuda").repeat_interleave(torch.ones_like(sc) << sc)
        perm = torch.argsort(graph.double() + 0.999 * torch.rand(n, device="cuda", generator=gen, dtype=torch.float64))
    else:
        perm = torch.randperm(n, device="cuda", generator=gen)
    return perm[src], perm[dst], n, first


def _road_edges(width, drop, gen):
    """4-neighbour lattice, the share `drop` of its edges dropped, plus 0.5 % as many random long edges."""
    ids = torch.arange(width * width, device="cuda", dtype=torch.int64).view(width, width)
    src = torch.cat([ids[:, :-1].reshape(-1), ids[:-1, :].reshape(-1)])
    dst = torch.cat([ids[:, 1:].reshape(-1), ids[1:, :].reshape(-1)])
    keep = torch.rand(src.numel(), device="cuda", generator=gen) >= drop
    src, dst = src[keep], dst[keep]
    far = torch.randint(0, width * width, (2, max(1, int(0.005 * src.numel()))), device="cuda", generator=gen)
    return torch.cat([src, far[0]]), torch.cat([dst, far[1]]), width * width


def _csr(case, seed):
    """(row offsets, columns, sources of the edges, vertices, first vertex of each graph) on the GPU."""
    gen = _generator(seed)
    first = None
    if case["graph"] == "road":
        # components are asked for where streets are cut off: then more edges are missing
        src, dst, n = _road_edges(case["size"], 0.35 if case["op"] == "cc" else 0.02, gen)
    elif case["graph"] == "batch":
        scales = np.random.default_rng(int(seed)).permutation(10 + np.arange(case["size"]) % 7).tolist()
        src, dst, n, first = _rmat_edges(scales, case["ef"], gen)
    else:
        src, dst, n, _ = _rmat_edges([case["size"]], case["ef"], gen)
    n += case["extra"]
    keep = src != dst
    src, dst = src[keep], dst[keep]
    if case["graph"] != "rmat_dir":
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    key = torch.unique(src * n + dst)
    if case["op"] == "ppr":  # a gradient per edge: every seed's graph keeps the same number of them
        key = key[torch.randperm(key.numel(), device="cuda", generator=gen)[:int(_kept(case) * case["ef"] * n)]]
        key = torch.sort(key).values
    src, dst = key // n, key % n
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    return off, dst, src, n, first


def _weights(src, dst, wmax, seed):
    """Symmetric integer weights in [1, wmax]: a hash of the unordered pair and the seed."""
    x = torch.minimum(src, dst) * 0x1000193 ^ torch.maximum(src, dst) * 0x9E3779B1 ^ (int(seed) * 0x85EBCA6B & 0x7FFFFFFF)
    x = (x ^ (x >> 15)) * 0x2C1B3C6D & 0x7FFFFFFFFFFF
    x = (x ^ (x >> 12)) * 0x297A2D39 & 0x7FFFFFFFFFFF
    return (x ^ (x >> 15)) % wmax + 1


def _sources(case, off, first, seed):
    """Seeded vertices that have edges (distinct); the hub when one graph of a batch or a host call asks for it."""
    deg = off[1:] - off[:-1]
    if case["op"] == "bfs_host":
        return np.array([int(torch.argmax(deg))], np.int32)
    if case["op"] == "bfs_batch":
        f = first.tolist()
        return np.array([int(torch.argmax(deg[f[i]:f[i + 1]])) for i in range(len(f) - 1)], np.int32)
    cand = torch.nonzero(deg > 0).reshape(-1)
    pick = torch.randperm(cand.numel(), device="cuda", generator=_generator(int(seed) + 77))[:case["nsrc"]]
    return cand[pick].to(torch.int32).cpu().numpy()


def _ppr_inputs(case, off, src, n, seed):
    """Row-normalised lognormal edge weights, sparse teleport distributions, and the loss's weights."""
    gen = _generator(int(seed) + 5)
    w = torch.exp(torch.randn(src.numel(), device="cuda", generator=gen, dtype=torch.float64))
    w = w / torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, src, w)[src]
    t = torch.zeros((n, case["nvec"]), device="cuda")
    k = min(100, n)
    for c in range(case["nvec"]):
        t[torch.randperm(n, device="cuda", generator=gen)[:k], c] = 1.0 / k
    return w.float(), t, torch.randn((n, case["nvec"]), device="cuda", generator=gen)


def prepare(case, seed):
    off, col, src, n, first = _csr(case, seed)
    host = gg.HostGraph(off.to(torch.int32).cpu().numpy(), col.to(torch.int32).cpu().numpy(),
                        directed=case["graph"] == "rmat_dir")
    if case["wmax"]:
        host.edge_values = _weights(src, col, case["wmax"], seed).to(torch.int32).cpu().numpy()
    if first is not None:
        host.graph_offsets = first.cpu().numpy()
    st = dict(case=case, graph=gg.Graph(host))
    op = case["op"]
    if op == "ppr":
        w, t, c = _ppr_inputs(case, off, src, n, seed)
        st.update(w=w.requires_grad_(True), t=t.requires_grad_(True), c=c)
    else:
        if op not in ("cc", "pagerank"):
            st["src"] = _sources(case, off, first, seed)
        rows = len(st["src"]) if op.endswith("_multi") else 1
        if op != "bfs_host":
            st["out"] = torch.empty((rows, n) if rows > 1 else (n,), device="cuda",
                                    dtype=torch.float32 if op == "pagerank" else torch.int32)
        if op == "bfs_pred":
            st["pred"] = torch.empty(n, dtype=torch.int32, device="cuda")
        more = dict(tolerance=1e-6, iter_num=100) if op == "pagerank" else {}
        st["opts"] = gg.default_options(outputs_on_device=1, compute_stats=0, **more)
    del off, col, src, first
    torch.cuda.empty_cache()  # the library allocates beside torch's pool
    return st


# -------------------------------------------------------------------- a pass --
def _call(status):
    if status:
        raise RuntimeError(gg.lib.mg_last_error().decode())


def run(state):
    g, op = state["graph"], state["case"]["op"]
    if op == "bfs_host":
        depths, stats = g.bfs(int(state["src"][0]))
        return {"depths": depths, "reached": stats["vertices_reached"], "edges": stats["edges_traversed"]}
    if op == "ppr":
        ranks = ppr(g, state["w"], state["t"])
        gw, gt = torch.autograd.grad((ranks * state["c"]).sum(), (state["w"], state["t"]))
        return {"ranks": ranks.detach(), "grad_weights": gw, "grad_teleport": gt}
    out, opts = state["out"], C.byref(state["opts"])
    if op in ("bfs", "sssp"):
        _call(getattr(gg.lib, "mg_" + op)(g.handle, int(state["src"][0]), out.data_ptr(), None, opts))
    elif op == "bfs_pred":
        pred = state["pred"]
        _call(gg.lib.mg_bfs_pred(g.handle, int(state["src"][0]), out.data_ptr(), pred.data_ptr(), None, opts))
        return {"depths": out, "pred": pred}
    elif op == "bfs_batch":
        _call(gg.lib.mg_bfs_batch(g.handle, state["src"].ctypes.data, out.data_ptr(), None, opts))
    elif op in ("bfs_roots", "bfs_multi", "sssp_multi"):
        src = state["src"]
        _call(getattr(gg.lib, "mg_" + op)(g.handle, src.ctypes.data, len(src), out.data_ptr(), None, opts))
    else:  # cc, pagerank
        _call(getattr(gg.lib, "mg_" + op)(g.handle, out.data_ptr(), None, opts))
    return out


# ------------------------------------------------- what a pass cannot do without --
def _kept(case):
    """Share of the drawn R-MAT edges that are neither self-loops nor duplicates, at least."""
    return 0.93 if case["size"] >= 18 else 0.85 if case["size"] >= 14 else 0.5


def _size(case):
    """(vertices, stored edges) of the case's graphs, about."""
    if case["graph"] == "road":
        return case["size"] ** 2, 3.94 * case["size"] ** 2
    if case["graph"] == "batch":
        n = case["size"] * (2 ** 17 - 2 ** 10) / 7
        return n, 2 * 0.85 * case["ef"] * n
    n = 2.0 ** case["size"]
    return n + case["extra"], _kept(case) * case["ef"] * n * (1 if case["graph"] == "rmat_dir" else 2)


def work(case):
    """The graph (and its weights) read once, the results written once. PageRank and its
    personalised form multiply and add once per edge, column and pass over the graph, of which
    a solve needs about as many as are given here."""
    n, m = _size(case)
    op, nvec = case["op"], case["nvec"]
    graph = 4 * (n + 1) + 4 * m
    if op == "ppr":
        # graph and weights; teleport, loss weights; ranks and both gradients
        return {"bytes": graph + 8 * m + 16 * n * nvec, "flops": 2.0 * m * nvec * (2 * 60 + 1)}
    if op == "pagerank":
        return {"bytes": graph + 4 * n, "flops": 2.0 * m * 20}
    weights = 4 * m if case["wmax"] else 0
    results = case["nsrc"] if op.endswith("_multi") else (2 if op == "bfs_pred" else 1)
    return {"bytes": graph + weights + 4.0 * n * results}


def tolerance(case):
    if case["op"] == "pagerank":
        return {"rel": 2e-6}
    if case["op"] == "ppr":
        return {"rel": 2e-6}
    return "exact"


# ------------------------------------------------------- the same in 64 bits --
def _levels(n, src, dst, roots):
    d = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    d[roots] = 0
    level = 0
    while True:
        nxt = dst[d[src] == level]
        nxt = nxt[d[nxt] < 0]
        if nxt.numel() == 0:
            return d
        level += 1
        d[nxt] = level


def _distances(n, src, dst, w, root):
    d = torch.full((n,), UNREACHED_SSSP, dtype=torch.int64, device="cuda")
    d[root] = 0
    new = torch.zeros(n, dtype=torch.bool, device="cuda")
    new[root] = True
    while bool(new.any()):
        e = torch.nonzero(new[src]).reshape(-1)
        nd = d.clone().scatter_reduce_(0, dst[e], d[src[e]] + w[e], "amin")
        new = nd < d
        d = nd
    return d


def _components(n, src, dst):
    lab = torch.arange(n, device="cuda")
    while True:
        new = lab.clone().scatter_reduce_(0, dst, lab[src], "amin")
        new = torch.minimum(new, new[new])
        if torch.equal(new, lab):
            return lab
        lab = new


def _pagerank(n, src, dst, off, tol, iters):
    deg = (off[1:] - off[:-1]).double()
    inv = torch.where(deg > 0, 1.0 / deg.clamp(min=1), torch.zeros_like(deg))
    r = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    d = 0.85
    for _ in range(iters):
        base = (1 - d) / n + d * float(r[deg == 0].sum()) / n
        new = base + d * torch.zeros_like(r).index_add_(0, dst, (r * inv)[src])
        done = float((new - r).abs().sum()) <= tol
        r = new
        if done:
            break
    return r


def _ppr_solve(mat, rhs, alpha, d, tol):
    x, norm = rhs.clone(), float(rhs.abs().sum())
    for _ in range(10000):
        new = alpha * rhs + d * (mat @ x)
        change = float((new - x).abs().sum())
        x = new
        if change <= tol * norm:
            break
    return x


def _ppr(case, off, col, src, n, seed):
    w, t, c = (x.double() for x in _ppr_inputs(case, off, src, n, seed))
    d, tol = 0.85, 1e-7
    p = torch.sparse_csr_tensor(off, col, w, (n, n))
    order = torch.argsort(col, stable=True)
    toff = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    toff[1:] = torch.cumsum(torch.bincount(col, minlength=n), 0)
    ranks = _ppr_solve(torch.sparse_csr_tensor(toff, src[order], w[order], (n, n)), t, 1 - d, d, tol)
    lam = _ppr_solve(p, c, 1.0, d, tol)
    gw = torch.empty_like(w)
    for b in range(0, gw.numel(), 1 << 21):
        gw[b:b + (1 << 21)] = d * (lam[col[b:b + (1 << 21)]] * ranks[src[b:b + (1 << 21)]]).sum(1)
    return {"ranks": ranks, "grad_weights": gw, "grad_teleport": (1 - d) * lam}


def exact(case, seed):
    off, col, src, n, first = _csr(case, seed)
    op = case["op"]
    if op == "ppr":
        return _ppr(case, off, col, src, n, seed)
    if op == "cc":
        return _components(n, src, col)
    if op == "pagerank":
        return _pagerank(n, src, col, off, 1e-6, 100)
    roots = torch.from_numpy(_sources(case, off, first, seed)).long().cuda()
    if op in ("sssp", "sssp_multi"):
        w = _weights(src, col, case["wmax"], seed)
        rows = [_distances(n, src, col, w, s) for s in roots]
        return torch.stack(rows) if len(rows) > 1 else rows[0]
    if op == "bfs_multi":
        rows = [_levels(n, src, col, s) for s in roots]
        return torch.stack(rows) if len(rows) > 1 else rows[0]
    if op == "bfs_batch":
        roots = roots + first[:-1]
    d = _levels(n, src, col, roots)
    if op == "bfs_host":
        reached = d >= 0
        return {"depths": d, "reached": int(reached.sum()), "edges": int((off[1:] - off[:-1])[reached].sum())}
    if op == "bfs_pred":
        # the largest in-neighbour one level up, of reached vertices
        ok = (d[col] - d[src] == 1) & (d[src] >= 0)
        pred = torch.full((n,), -1, dtype=torch.int64, device="cuda")
        pred.scatter_reduce_(0, col[ok], src[ok], "amax")
        return {"depths": d, "pred": pred}
    return d
