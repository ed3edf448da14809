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
