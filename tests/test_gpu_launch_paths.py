"""GPU parity at the edges of the launch rules: one-launch and level-by-level
traversals, edge bounds of the batched SSSP, row widths of the personalised
PageRank solve."""
import numpy as np
import pytest

import oracle
from gpugraph_b200 import Graph, HostGraph, MapGraphError, _lib

pytestmark = pytest.mark.gpu

DIRS = [_lib.MG_DIR_AUTO, _lib.MG_DIR_PUSH, _lib.MG_DIR_PULL]


def star(n, arms=1):
    """Vertex 0 joined to every other one (its adjacency spans many queue entries), plus `arms` paths of 3."""
    edges = [(0, v) for v in range(1, n)]
    for a in range(arms):
        b = n + 3 * a
        edges += [(a + 1, b), (b, b + 1), (b + 1, b + 2)]
    m = n + 3 * arms
    src, dst = np.array(edges).T
    src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    order = np.lexsort((dst, src))
    ro = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=m))]).astype(np.int32)
    return HostGraph(ro, dst[order].astype(np.int32), None)


def padded(hg, k):
    """hg with k isolated vertices appended."""
    ro = np.concatenate([hg.row_offsets, np.full(k, hg.row_offsets[-1], np.int32)])
    return HostGraph(ro, hg.column_indices, hg.edge_values, hg.directed)


# one vertex; a word of vertices and one more; a hub of 255, 256, 257 and 5000 edges (entries hold 256);
# many levels; a dense graph; a vertex count that is no multiple of 32 or 4
GRAPHS = {
    "one": lambda: HostGraph(np.array([0, 0], np.int32), np.zeros(0, np.int32)),
    "star33": lambda: star(33),
    "star256": lambda: star(256, 2),
    "star257": lambda: star(257, 2),
    "star258": lambda: star(258, 2),
    "star5001": lambda: star(5001, 40),
    "road": lambda: HostGraph.road_grid(90, 0.02, 0.0, seed=3),
    "rmat": lambda: HostGraph.rmat(13, 16, seed=9),
    "rmat_odd": lambda: padded(HostGraph.rmat(12, 8, seed=5), 3),
    "directed": lambda: HostGraph.rmat(12, 8, seed=6, symmetrize=False),
}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_bfs_one_launch_equals_level_loop(name):
    hg = GRAPHS[name]()
    g = Graph(hg, directed=name == "directed")
    deg = hg.out_degree()
    for s in sorted({0, hg.nodes - 1, int(np.argmax(deg))}):
        ref = oracle.bfs(hg.row_offsets, hg.column_indices, s)
        reached = ref >= 0
        for d in DIRS:
            for mode in ({}, dict(use_cuda_graph=0), dict(ordered_frontier=1), dict(alpha=1e9, beta=0.5)):
                out, st = g.bfs(s, direction=d, **mode)
                assert np.array_equal(out, ref), (s, d, mode)
                assert st["vertices_reached"] == int(reached.sum())
                assert st["edges_traversed"] == int(deg[reached].sum())
                assert st["iterations"] == int(ref.max()) + 1 and st["converged"] == 1
                assert st["push_iterations"] + st["pull_iterations"] == st["iterations"]
        for cap in (0, 1, 2):
            a, sa = g.bfs(s, iter_num=cap)
            b, sb = g.bfs(s, iter_num=cap, use_cuda_graph=0)
            assert np.array_equal(a, b) and sa["iterations"] == sb["iterations"]
            assert sa["converged"] == sb["converged"] and sa["vertices_reached"] == sb["vertices_reached"]


def test_bfs_one_launch_roots_and_interleaved_runs():
    # several roots (more than a warp), other algorithms between runs, and runs on another stream
    torch = pytest.importorskip("torch")
    hg = HostGraph.rmat(13, 8, seed=31).with_weights(1, 9, seed=1)
    g = Graph(hg)
    rng = np.random.default_rng(0)
    side = torch.cuda.Stream()
    for k in (2, 31, 32, 33, 700):
        roots = rng.choice(hg.nodes, k, replace=False).astype(np.int32)
        ref = np.stack([oracle.bfs(hg.row_offsets, hg.column_indices, r) for r in roots[:40]])
        out, _ = g.bfs_roots(roots[:40])
        best = np.where(ref >= 0, ref, 1 << 30).min(0)
        assert np.array_equal(out, np.where(best < 1 << 30, best, -1)), k
        g.cc()
        a, _ = g.bfs(int(roots[0]), stream=side.cuda_stream)
        assert np.array_equal(a, ref[0])
        g.sssp(int(roots[0]))


@pytest.mark.parametrize("nsrc", [1, 2, 33, 64])
@pytest.mark.parametrize("kind", ["skewed", "directed", "islands"])
def test_sssp_multi_edge_bounds(kind, nsrc):
    # skewed enough that the bounds are kept; with a source that never reaches the hub ("islands",
    # "directed") they must stay off, without it they prune from the level every source reached the hub
    hg = HostGraph.rmat(14, 4, seed=17, symmetrize=kind != "directed")
    if kind == "islands":
        hg = padded(hg, 5)
    hg = hg.with_weights(1, 64, seed=3)
    indeg = np.bincount(hg.column_indices, minlength=hg.nodes)
    assert indeg.max() > 64 * max(1.0, hg.edges / hg.nodes)
    g = Graph(hg, directed=kind == "directed")
    rng = np.random.default_rng(nsrc)
    srcs = rng.choice(np.flatnonzero(hg.out_degree() > 0), nsrc, replace=False).astype(np.int32)
    if kind == "islands":
        srcs[-1] = hg.nodes - 1
    for mode in ({}, dict(use_cuda_graph=0)):
        out, _ = g.sssp_multi(srcs, **mode)
        for k, s in enumerate(srcs):
            assert np.array_equal(out[k], oracle.sssp(hg.row_offsets, hg.column_indices, hg.edge_values, s)), k


D = 0.85


def _ppr_case(nvec, seed=7, scale=9):
    hg = HostGraph.rmat(scale, 16, seed=seed, symmetrize=False)
    rng = np.random.default_rng(seed)
    src = np.repeat(np.arange(hg.nodes), np.diff(hg.row_offsets))
    w = rng.lognormal(0.0, 1.0, size=hg.edges)
    w = w / np.bincount(src, weights=w, minlength=hg.nodes)[src]
    t = np.zeros((hg.nodes, nvec))
    for c in range(nvec):
        t[rng.choice(hg.nodes, size=20, replace=False), c] = 0.05
    return hg, src, w, t, rng.standard_normal((hg.nodes, nvec))


def _ppr_dense(torch, hg, src, w, t, c):
    w64, t64 = torch.tensor(w, requires_grad=True), torch.tensor(t, requires_grad=True)
    p = torch.zeros((hg.nodes, hg.nodes), dtype=torch.float64).index_put(
        (torch.as_tensor(src), torch.as_tensor(hg.column_indices.astype(np.int64))), w64, accumulate=True)
    r = torch.linalg.solve(torch.eye(hg.nodes, dtype=torch.float64) - D * p.T, (1 - D) * t64)
    (r * torch.tensor(c)).sum().backward()
    return r.detach(), w64.grad, t64.grad


def _ppr_check(torch, g, hg, src, w, t, c):
    from gpugraph_b200.ppr import ppr

    ref_r, ref_w, ref_t = _ppr_dense(torch, hg, src, w, t, c)
    wt = torch.tensor(w, dtype=torch.float32, device="cuda", requires_grad=True)
    tt = torch.tensor(t, dtype=torch.float32, device="cuda", requires_grad=True)
    r = ppr(g, wt, tt)
    (r * torch.tensor(c, dtype=torch.float32, device="cuda")).sum().backward()
    # the solve stops at an L1 change of 1e-7 of its right-hand side, d/(1-d) = 5.7 times that is left;
    # sums of FP32 products of this size add about 1e-6: the bounds of the other PPR tests
    assert (r.detach().double().cpu() - ref_r).abs().sum(0).max() < 2e-5
    assert (wt.grad.double().cpu() - ref_w).norm() / ref_w.norm() < 1e-4
    assert (tt.grad.double().cpu() - ref_t).norm() / ref_t.norm() < 1e-4


@pytest.mark.parametrize("nvec", [1, 3, 4, 5, 8, 9, 16, 17, 32, 33, 61, 64])
def test_ppr_every_row_width(nvec):
    # 1, 2, 4, 8 and 16 lanes per list, with and without padding columns
    torch = pytest.importorskip("torch")
    hg, src, w, t, c = _ppr_case(nvec)
    _ppr_check(torch, Graph(hg, directed=True), hg, src, w, t, c)


def test_ppr_width_grows_and_shrinks_on_one_graph():
    # the workspace is replaced when the rows get wider; a narrower solve after that must use the new one
    torch = pytest.importorskip("torch")
    hg, *_ = _ppr_case(4)
    g = Graph(hg, directed=True)
    for nvec in (4, 32, 4, 7, 64, 32, 1):
        _, src, w, t, c = _ppr_case(nvec)
        _ppr_check(torch, g, hg, src, w, t, c)


@pytest.mark.parametrize("length", [0, 1, 7, 8, 9, 255, 256, 257, 513])
def test_ppr_list_lengths(length):
    # one vertex with `length` in-edges and out-edges: the steps of 8, the chunks of 256 and what is left over
    torch = pytest.importorskip("torch")
    n = 600
    edges = {(v, 0) for v in range(1, length + 1)} | {(0, v) for v in range(20, length + 20)}
    edges |= {(v, v % 19 + 1) for v in range(1, 40)}
    src, dst = np.array(sorted(edges)).T
    ro = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    hg = HostGraph(ro, dst.astype(np.int32), None, directed=True)
    rng = np.random.default_rng(length)
    w = rng.uniform(0.1, 1.0, size=hg.edges)
    w = w / np.bincount(src, weights=w, minlength=n)[src]
    t = np.zeros((n, 12))
    for c in range(12):
        t[rng.choice(n, 30, replace=False), c] = 1 / 30
    t[0] += 0.1
    _ppr_check(torch, Graph(hg, directed=True), hg, src, w, t, rng.standard_normal((n, 12)))


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("lo,hi", [(0, 0), (1, 1), (0, 3), (1, 64), (1, 1000), (50_000, 90_000)])
def test_sssp_one_launch_equals_level_loop(name, lo, hi):
    # windows of one weight and of many, zero weights, sums past the unreachable distance (100000000)
    hg = GRAPHS[name]().with_weights(lo, hi, seed=2)
    g = Graph(hg, directed=name == "directed")
    for s in sorted({0, hg.nodes - 1, hg.max_degree_vertex()}):
        ref = oracle.sssp(hg.row_offsets, hg.column_indices, hg.edge_values, s)
        out, st = g.sssp(s)
        assert np.array_equal(out, ref) and st["converged"] == 1, s
        assert st["vertices_reached"] == int((ref < 100000000).sum())
        host, _ = g.sssp(s, use_cuda_graph=0)
        assert np.array_equal(host, ref), s


@pytest.mark.parametrize("name", list(GRAPHS))
def test_cc_labels_at_the_edges(name):
    hg = GRAPHS[name]()
    if name == "directed":
        pytest.skip("union-find serves symmetric graphs")
    g = Graph(hg)
    ref, _ = g.cc(generic_engine=1)
    for _ in range(5):
        assert np.array_equal(g.cc()[0], ref)
    # lists in any order: the first neighbour need not be the smallest
    col = hg.column_indices.copy()
    for v in range(hg.nodes):
        b, e = hg.row_offsets[v], hg.row_offsets[v + 1]
        col[b:e] = col[b:e][::-1]
    assert np.array_equal(Graph(HostGraph(hg.row_offsets, col, None)).cc()[0], ref)


def _lists(lengths, n):
    """Directed graph whose vertex i has lengths[i] in-edges from distinct vertices; the rest feed vertex 0 in a ring."""
    edges = set()
    for i, k in enumerate(lengths):
        edges |= {((i + 1 + j) % n, i) for j in range(k)}
    edges |= {(v, (v + 1) % n) for v in range(len(lengths), n, 2)}
    src, dst = np.array(sorted(edges)).T
    ro = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    return HostGraph(ro, dst.astype(np.int32), None, directed=True)


def test_pagerank_list_lengths_and_loops():
    # in-lists around the lane-serial (8), chunk (128, 1024) limits; one launch and level loop
    hg = _lists([0, 1, 7, 8, 9, 31, 127, 128, 129, 1023, 1024, 1025, 1152, 1153, 3000], 4001)
    g = Graph(hg, directed=True)
    t = hg.transpose()
    for iters in (0, 1, 2, 25):
        a, sa = g.pagerank(iter_num=iters, tolerance=0.0)
        b, sb = g.pagerank(iter_num=iters, tolerance=0.0, use_cuda_graph=0)
        ref, _, _ = oracle.pagerank_fp64(hg.row_offsets, t.row_offsets, t.column_indices, 0.85, 0.0, iters)
        assert sa["iterations"] == sb["iterations"] == iters
        assert np.abs(a - ref).sum() < 1e-6 and np.abs(b - ref).sum() < 1e-6  # the FP32 bound of the other tests


@pytest.mark.parametrize("scale,ef", [(18, 16), (20, 17)])
def test_pagerank_renumbered_graph_both_loops(scale, ef):
    # below and above the size up to which a solve is one launch, each also through the host-driven loop
    hg = HostGraph.rmat(scale, ef, seed=8, symmetrize=False)
    g = Graph(hg, directed=True)
    t = hg.transpose()
    for mode in ({}, dict(use_cuda_graph=0)):
        r, st = g.pagerank(tolerance=1e-7, iter_num=60, **mode)
        ref, _, _ = oracle.pagerank_fp64(hg.row_offsets, t.row_offsets, t.column_indices, 0.85, 0.0,
                                         int(st["iterations"]))
        assert np.abs(r - ref).sum() < 1e-6


def test_one_launch_calls_from_several_threads():
    # each thread has its own graph and stream; the calls overlap in time
    torch = pytest.importorskip("torch")
    import threading

    hgs = [HostGraph.rmat(13, 8, seed=50 + i).with_weights(1, 20, seed=i) for i in range(4)]
    refs = [(oracle.bfs(h.row_offsets, h.column_indices, 1), oracle.sssp(h.row_offsets, h.column_indices,
                                                                        h.edge_values, 1)) for h in hgs]
    bad = []

    def work(i):
        try:
            g, st = Graph(hgs[i]), torch.cuda.Stream()
            lab = g.cc()[0]
            for _ in range(25):
                ok = np.array_equal(g.bfs(1, stream=st.cuda_stream)[0], refs[i][0])
                ok &= np.array_equal(g.sssp(1, stream=st.cuda_stream)[0], refs[i][1])
                ok &= np.array_equal(g.cc(stream=st.cuda_stream)[0], lab)
                g.pagerank(stream=st.cuda_stream, iter_num=5)
                if not ok:
                    bad.append(i)
        except Exception as e:  # reported by the main thread
            bad.append(repr(e))

    th = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad


@pytest.mark.parametrize("name", list(GRAPHS) + ["long_lists"])
def test_bfs_multi_one_launch_equals_level_loop(name):
    # levels before and past the 16 of the level stack, both directions and runs that flip between them
    # (alpha_multi, beta), lists with and without ranges, duplicated sources, limited runs
    # long_lists: in-lists past 512 edges and more found vertices in a level than get their ranges at once
    hg = HostGraph.rmat(18, 8, seed=3) if name == "long_lists" else GRAPHS[name]()
    g = Graph(hg, directed=name == "directed")
    deg = hg.out_degree()
    rng = np.random.default_rng(4)
    for nsrc in (1, 33, 64):
        srcs = rng.integers(0, hg.nodes, nsrc).astype(np.int32)
        srcs[0] = hg.max_degree_vertex()
        some = {int(s): oracle.bfs(hg.row_offsets, hg.column_indices, int(s)) for s in srcs[:6]}
        host, _ = g.bfs_multi(srcs, use_cuda_graph=0)
        reached = host >= 0
        for d in DIRS:
            for mode in ({}, dict(alpha_multi=1e9, beta=0.5), dict(alpha_multi=1e-9, beta=1e9)):
                out, st = g.bfs_multi(srcs, direction=d, **mode)
                assert np.array_equal(out, host), (nsrc, d, mode)
                assert st["vertices_reached"] == int(reached.sum()) and st["converged"] == 1
                assert st["edges_traversed"] == int((reached * deg[None, :]).sum())
        for k, s in enumerate(srcs):
            if int(s) in some:
                assert np.array_equal(host[k], some[int(s)])


def _dag(n, deg, hub, lo, hi, seed):
    """Directed acyclic graph, edges from lower to higher ids, int32 weights in [lo, hi]; vertex `hub` (if any) is
    a head of every lower one. Distances by one pass over the vertices in order."""
    rng = np.random.default_rng(seed)
    src = np.repeat(np.arange(n - 1), deg)
    dst = src + 1 + (rng.random(src.size) * np.minimum(60, n - 1 - src)).astype(np.int64)
    if hub:
        src, dst = np.concatenate([src, np.arange(hub)]), np.concatenate([dst, np.full(hub, hub)])
    key = np.unique(src * n + dst)
    src, dst = key // n, key % n
    ro = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    w = rng.integers(lo, hi, src.size, endpoint=True)
    hg = HostGraph(ro, dst.astype(np.int32), w.astype(np.int32), directed=True)

    def dists(srcs):
        d = np.full((n, len(srcs)), 100000000, np.int64)
        d[srcs, np.arange(len(srcs))] = 0
        for u in range(n):
            b, e = ro[u], ro[u + 1]
            cand = np.where(d[u] < 100000000, d[u] + w[b:e, None], 100000000)
            d[dst[b:e]] = np.minimum(d[dst[b:e]], cand)
        return d.T

    return hg, dists


@pytest.mark.parametrize("hub,nsrc,deg", [(0, 56, 12), (0, 57, 12), (0, 64, 12), (0, 57, 5), (0, 64, 5),
                                          (1500, 9, 5), (1500, 37, 5), (1500, 64, 12)])
@pytest.mark.parametrize("lo,hi", [(-40, 60), (-40, -1), (0, 7)])
def test_sssp_multi_sources_that_do_not_reach_each_other(hub, nsrc, deg, lo, hi):
    # (5 and 12 edges a vertex: edges relaxed by lanes and by rows, also with 57 sources on flat graphs)
    # most sources cannot reach the early vertices, many are active on one edge: a source that has not reached a
    # tail must stay unreached at the head, also where the weight is negative (100000000 + w < 100000000)
    hg, dists = _dag(2000, deg, hub, lo, hi, seed=nsrc)
    srcs = np.sort(np.random.default_rng(1).choice(hub or 1900, nsrc, replace=False)).astype(np.int32)
    ref = dists(srcs)
    assert (ref == 100000000).mean() > 0.2
    g = Graph(hg)
    for mode in ({}, dict(use_cuda_graph=0)):
        out, st = g.sssp_multi(srcs, **mode)
        assert np.array_equal(out, ref)
        assert st["converged"] == 1 and st["vertices_reached"] == int((ref != 100000000).sum())
    assert np.array_equal(g.sssp(int(srcs[0]))[0], ref[0])


@pytest.mark.parametrize("nsrc", [1, 15, 37, 64])
def test_sssp_weights_whose_sums_wrap(nsrc):
    # d + w past the int range gives a negative distance. On a tree every vertex has one path, so its distance is
    # defined all the same; edge bounds (the last vertex is a sink that all others point to, so the graph is skewed)
    # and windows rely on distances in [0, 100000000] and must not be used
    n, inf = 3000, 100000000
    rng = np.random.default_rng(nsrc)
    v = np.arange(1, n - 1)
    par = v - 1 - (rng.random(v.size) * np.minimum(6, v)).astype(np.int64)
    w = rng.integers(1, 50, v.size)
    w[rng.random(v.size) < 0.05] = 2147483640
    src, dst, wt = np.concatenate([par, np.arange(n - 1)]), np.concatenate([v, np.full(n - 1, n - 1)]), np.concatenate(
        [w, np.ones(n - 1, np.int64)])
    order = np.lexsort((dst, src))
    ro = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    hg = HostGraph(ro, dst[order].astype(np.int32), wt[order].astype(np.int32), directed=True)
    chain = [n - 2]  # the sources: its ancestors, top first, so that each of them reaches a long part of the tree
    while chain[-1]:
        chain.append(int(par[chain[-1] - 1]))
    srcs = np.array(chain[::-1][:nsrc], np.int32)
    ref = np.full((n - 1, nsrc), inf, np.int64)
    ref[srcs, np.arange(nsrc)] = 0
    for x in range(1, n - 1):
        d = ref[par[x - 1]]
        ref[x] = np.minimum(ref[x], np.where(d < inf, (d + w[x - 1]).astype(np.int32), inf))
    assert ref.min() < -2000000000
    g = Graph(hg)
    out, st = g.sssp_multi(srcs)
    assert np.array_equal(out[:, :-1], ref.T) and st["converged"] == 1
    for mode in ({}, dict(use_cuda_graph=0)):
        one, st = g.sssp(int(srcs[0]), **mode)
        assert np.array_equal(one[:-1], ref[:, 0]) and st["converged"] == 1


@pytest.mark.parametrize("shift", [0, 1, 2, 4])
def test_device_results_at_any_address(shift):
    # a kernel writes a device buffer itself where it is aligned; at an odd address the result is copied there
    torch = pytest.importorskip("torch")
    import ctypes as C

    from gpugraph_b200.ppr import ppr

    lib = _lib.lib
    hg = HostGraph.rmat(10, 8, seed=3).with_weights(1, 64, seed=1)
    hd = HostGraph.rmat(9, 8, seed=5, symmetrize=False)
    g, gd = Graph(hg), Graph(hd, directed=True)
    s, opts = hg.max_degree_vertex(), _lib.default_options(outputs_on_device=1)
    w = torch.tensor(1.0 / np.repeat(np.maximum(hd.out_degree(), 1), hd.out_degree()), dtype=torch.float32,
                     device="cuda")

    def result(call, n, dtype):
        buf = torch.full((4 * n + 8,), 0x55, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        _lib.check(call(buf.data_ptr() + shift), "call")
        h = buf.cpu().numpy()
        assert (h[:shift] == 0x55).all() and (h[shift + 4 * n:] == 0x55).all()
        return h[shift:shift + 4 * n].copy().view(dtype)

    o = C.byref(opts)
    n, nd = hg.nodes, hd.nodes
    ref = oracle.bfs(hg.row_offsets, hg.column_indices, s)
    assert np.array_equal(result(lambda p: lib.mg_bfs(g.handle, s, p, None, o), n, np.int32), ref)
    assert np.array_equal(result(lambda p: lib.mg_sssp(g.handle, s, p, None, o), n, np.int32), g.sssp(s)[0])
    assert np.array_equal(result(lambda p: lib.mg_cc(g.handle, p, None, o), n, np.int32), g.cc()[0])
    rank = result(lambda p: lib.mg_pagerank(gd.handle, p, None, o), nd, np.float32)
    assert np.abs(rank - gd.pagerank(iter_num=opts.iter_num)[0]).sum() < 1e-6
    opts.tolerance = 1e-7
    for nvec in (3, 4):
        tele = torch.zeros((nd, nvec), device="cuda")
        tele[::5] = 5.0 / nd
        torch.cuda.synchronize()
        r = result(lambda p: lib.mg_ppr_forward(gd.handle, w.data_ptr(), tele.data_ptr(), nvec, p, None, o), nd * nvec,
                   np.float32).reshape(nd, nvec)
        assert np.abs(r - ppr(gd, w, tele, max_iter=opts.iter_num).cpu().numpy()).max() < 1e-7


@pytest.mark.parametrize("leaves", [1 << 22, (1 << 22) + 1])
def test_bfs_in_list_too_long_for_a_barrier_wait(leaves):
    # a lane walks a pulled list: past 2^22 edges pulling calls go level by level, pushing ones stay in one launch
    n = leaves + 1
    ro = np.concatenate([[0], leaves + np.arange(n)]).astype(np.int32)
    g = Graph(HostGraph(ro, np.concatenate([np.arange(1, n), np.zeros(leaves)]).astype(np.int32)))
    ref = np.full(n, 2, np.int32)
    ref[0], ref[1] = 1, 0
    short = leaves <= 1 << 22
    for d, one in ((_lib.MG_DIR_PUSH, True), (_lib.MG_DIR_PULL, short), (_lib.MG_DIR_AUTO, short)):
        g.bfs(1, direction=d)
        _lib.lib.mg_kernel_launches(1)
        out, _ = g.bfs(1, direction=d)
        assert (_lib.lib.mg_kernel_launches(1) == 1) == one, d
        assert np.array_equal(out, ref)
    assert not g.cc()[0].any()


@pytest.mark.parametrize("mode", [{}, dict(use_cuda_graph=0)])
@pytest.mark.parametrize("nvec", [1, 2, 3, 7, 33])
def test_ppr_infinite_weight_in_padded_rows(nvec, mode):
    # an infinite weight makes its head's ranks infinite, and the solve stops when the change is no longer a number.
    # The padding columns of a row (0 times that weight) must not stop it earlier: a solve whose last columns repeat
    # up to a full row runs as many iterations and gives the same columns
    torch = pytest.importorskip("torch")
    import ctypes as C

    hd = HostGraph.rmat(9, 8, seed=5, symmetrize=False)
    g = Graph(hd, directed=True)
    w = 1.0 / np.repeat(np.maximum(hd.out_degree(), 1), hd.out_degree())
    w[hd.row_offsets[hd.max_degree_vertex()]] = np.inf
    w = torch.tensor(w, dtype=torch.float32, device="cuda")
    full = torch.rand((hd.nodes, nvec), device="cuda", generator=torch.Generator("cuda").manual_seed(1)) + 0.1
    full = torch.cat([full, full[:, -1:].expand(-1, -nvec % 4)], 1)
    got = []
    for k in (nvec, full.shape[1]):
        t = full[:, :k].contiguous()
        r, gt, gw = torch.empty_like(t), torch.empty_like(t), torch.empty_like(w)
        st, o = _lib.Stats(), _lib.default_options(tolerance=1e-7, iter_num=50, **mode)
        torch.cuda.synchronize()
        _lib.check(_lib.lib.mg_ppr_forward(g.handle, w.data_ptr(), t.data_ptr(), k, r.data_ptr(), C.byref(st),
                                           C.byref(o)), "forward")
        it = st.iterations
        _lib.check(_lib.lib.mg_ppr_backward(g.handle, w.data_ptr(), r.data_ptr(), t.data_ptr(), k, gw.data_ptr(),
                                            gt.data_ptr(), C.byref(st), C.byref(o)), "backward")
        got.append((it, st.iterations, r[:, :nvec].cpu().numpy(), gt[:, :nvec].cpu().numpy()))
    assert got[0][:2] == got[1][:2] and got[0][0] >= 2
    assert np.isinf(got[0][2]).any()
    assert np.array_equal(got[0][2], got[1][2], equal_nan=True)
    assert np.array_equal(got[0][3], got[1][3], equal_nan=True)


@pytest.mark.parametrize("kind,by_bfs", [("200 leaves", False), ("40000 leaves", False), ("wheel", True)])
def test_cc_hub_beside_a_lattice(kind, by_bfs):
    # a hub with few of the edges, or with many but not in the large component, says nothing about that (sampling
    # rounds); one joined to every vertex finds it
    grid = HostGraph.road_grid(150, 0.3, 0.0, seed=5)
    n = grid.nodes
    leaves = 0 if kind == "wheel" else int(kind.split()[0])
    b = 1 + np.arange(n - 1) if kind == "wheel" else n + np.arange(leaves)
    a = np.zeros(b.size, np.int64)
    src = np.concatenate([np.repeat(np.arange(n), np.diff(grid.row_offsets)), a, b])
    dst = np.concatenate([grid.column_indices, b, a])
    order = np.lexsort((dst, src))
    ro = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n + leaves))]).astype(np.int32)
    g = Graph(HostGraph(ro, dst[order].astype(np.int32)))
    ref, _ = g.cc(generic_engine=1)
    assert np.array_equal(g.cc()[0], ref)
    _lib.lib.mg_selftest_loops(_lib.MG_LOOP_TEST_WAITS)  # the BFS's barriers give up; the sampling has none
    try:
        if by_bfs:
            with pytest.raises(MapGraphError):
                g.cc()
        else:
            assert np.array_equal(g.cc()[0], ref)
    finally:
        _lib.lib.mg_selftest_loops(_lib.MG_LOOP_TEST_OFF)
    assert np.array_equal(g.cc()[0], ref)


@pytest.mark.parametrize("kind", ["path", "reversed path", "lattice", "combs", "two lattices"])
def test_cc_long_chains(kind):
    # graphs whose first neighbours chain up; ids in order, reversed and shuffled
    n = 1 << 15
    if kind.endswith("path"):
        a, b = np.arange(n - 1), np.arange(1, n)
    else:
        ids = np.arange(n).reshape(256, 128)
        a, b = ids[:-1].ravel(), ids[1:].ravel()
        rows = ids if kind == "lattice" else ids[:1] if kind == "combs" else np.concatenate([ids[:100], ids[101:]])
        a, b = np.concatenate([a, rows[:, :-1].ravel()]), np.concatenate([b, rows[:, 1:].ravel()])
        if kind == "two lattices":
            keep = (a // 128 != 100) & (b // 128 != 100)
            a, b = a[keep], b[keep]
    if kind == "reversed path":
        a, b = n - 1 - a, n - 1 - b
    for perm in (np.arange(n), np.random.default_rng(2).permutation(n)):
        src, dst = np.concatenate([perm[a], perm[b]]), np.concatenate([perm[b], perm[a]])
        order = np.lexsort((dst, src))
        ro = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
        g = Graph(HostGraph(ro, dst[order].astype(np.int32)))
        ref = oracle.cc(ro, dst[order].astype(np.int32))
        for _ in range(3):
            assert np.array_equal(g.cc()[0], ref)


@pytest.mark.parametrize("parts", [1, 2, 3, 9])
def test_cc_route_follows_what_the_bfs_reached(parts):
    # equal R-MAT graphs side by side: the hub's one holds 1/parts of the edges
    one = HostGraph.rmat(11, 16, seed=4)
    n, m = one.nodes, one.edges
    ro = np.concatenate([[0], (one.row_offsets[1:] + m * np.arange(parts)[:, None]).ravel()]).astype(np.int32)
    col = (one.column_indices + n * np.arange(parts)[:, None]).ravel().astype(np.int32)
    sub, reached = oracle.cc(one.row_offsets, one.column_indices), oracle.bfs(
        one.row_offsets, one.column_indices, one.max_degree_vertex())
    share = one.out_degree()[reached >= 0].sum() / (parts * m)
    by_bfs = share >= 0.8
    assert by_bfs == (parts == 1)
    ref = (sub + n * np.arange(parts)[:, None]).ravel()
    g = Graph(HostGraph(ro, col))
    for _ in range(3):
        assert np.array_equal(g.cc()[0], ref)
    _lib.lib.mg_selftest_loops(_lib.MG_LOOP_TEST_WAITS)
    try:
        if by_bfs:
            with pytest.raises(MapGraphError):
                g.cc()
        else:
            assert np.array_equal(g.cc()[0], ref)
    finally:
        _lib.lib.mg_selftest_loops(_lib.MG_LOOP_TEST_OFF)
    assert np.array_equal(g.cc()[0], ref)


@pytest.mark.parametrize("n", [(3 << 22) - 1, 3 << 22, (3 << 22) + 77])
@pytest.mark.parametrize("hi,graph", [(1, "rmat"), (1000, "rmat"), (64, "road"), (1000, "road")])
def test_sssp_sparse_ids_in_a_wide_graph(n, hi, graph):
    # a graph spread over n ids: from 3 * 2^22 on the selection looks only into the 256-vertex blocks where one may wait
    small = (HostGraph.rmat(12, 8, seed=7) if graph == "rmat" else HostGraph.road_grid(70, 0.05, 0.0, seed=7))
    small = small.with_weights(1, hi, seed=3)
    ids = np.sort(np.random.default_rng(5).choice(n, small.nodes, replace=False))
    ids[-1] = n - 1
    deg = np.zeros(n, np.int64)
    deg[ids] = small.out_degree()
    ro = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    g = Graph(HostGraph(ro, ids[small.column_indices].astype(np.int32), small.edge_values))
    for s in (small.max_degree_vertex(), small.nodes - 1):
        ref = np.full(n, 100000000, np.int32)
        ref[ids] = oracle.sssp(small.row_offsets, small.column_indices, small.edge_values, s)
        for _ in range(2):
            out, st = g.sssp(int(ids[s]))
            assert np.array_equal(out, ref) and st["converged"] == 1
