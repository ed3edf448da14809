"""GPU parity at the edges of the launch rules: one-launch and level-by-level
traversals, edge bounds of the batched SSSP, row widths of the personalised
PageRank solve."""
import numpy as np
import pytest

import oracle
from gpugraph_b200 import Graph, HostGraph, _lib

pytestmark = pytest.mark.gpu

DIRS = [_lib.MG_DIR_AUTO, _lib.MG_DIR_PUSH, _lib.MG_DIR_PULL]


def padded(hg, k):
    """hg with k isolated vertices appended."""
    ro = np.concatenate([hg.row_offsets, np.full(k, hg.row_offsets[-1], np.int32)])
    return HostGraph(ro, hg.column_indices, hg.edge_values, hg.directed)


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
