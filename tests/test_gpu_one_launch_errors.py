"""The calls that run in one cooperative launch, when something goes wrong on the way: the status they return, and
that the next call on the same graph is exact. The failures are made on the host; nothing faults or hangs."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

import oracle
from gpugraph_b200 import Graph, HostGraph, MapGraphError, _lib, concat_graphs

pytestmark = pytest.mark.gpu


class Calls:
    """A graph per kind of call (each with the call's reference result)."""

    def __init__(self):
        torch = pytest.importorskip("torch")
        from gpugraph_b200.ppr import ppr

        hg = HostGraph.rmat(12, 8, seed=31).with_weights(1, 64, seed=1)
        g = Graph(hg)
        s = hg.max_degree_vertex()
        srcs = np.random.default_rng(0).choice(hg.nodes, 33, replace=False).astype(np.int32)
        bfs = {int(v): oracle.bfs(hg.row_offsets, hg.column_indices, int(v)) for v in [s, *srcs]}
        sssp = oracle.sssp(hg.row_offsets, hg.column_indices, hg.edge_values, s)
        nearest = np.stack([np.where(bfs[int(v)] < 0, 1 << 30, bfs[int(v)]) for v in srcs]).min(0)
        nearest[nearest == 1 << 30] = -1
        labels, _ = g.cc(generic_engine=1)
        parts = [HostGraph.rmat(8, 8, seed=i) for i in range(3)]
        gb = Graph(concat_graphs(parts))
        batch = np.concatenate([oracle.bfs(p.row_offsets, p.column_indices, p.max_degree_vertex()) for p in parts])
        local = [p.max_degree_vertex() for p in parts]
        hd = HostGraph.rmat(10, 8, seed=5, symmetrize=False)
        gd = Graph(hd, directed=True)
        t = hd.transpose()
        rank = oracle.pagerank_fp64(hd.row_offsets, t.row_offsets, t.column_indices, 0.85, 0.0, 20)[0]
        w = torch.tensor(1.0 / np.repeat(np.maximum(hd.out_degree(), 1), hd.out_degree()), dtype=torch.float32,
                         device="cuda", requires_grad=True)
        tele = torch.zeros((hd.nodes, 4), device="cuda", requires_grad=True)
        with torch.no_grad():
            tele[::7] = 7.0 / hd.nodes
        host = ppr(gd, w, tele, use_cuda_graph=0).detach()

        def check_ppr():
            r = ppr(gd, w, tele)
            torch.autograd.grad(r.sum(), (w, tele))
            return (r.detach() - host).abs().max() < 1e-6

        self.calls = {
            "bfs": lambda: np.array_equal(g.bfs(s)[0], bfs[s]),
            "bfs_pred": lambda: np.array_equal(g.bfs_pred(s)[0], bfs[s]),
            "bfs_roots": lambda: np.array_equal(g.bfs_roots(srcs)[0], nearest),
            "bfs_batch": lambda: np.array_equal(gb.bfs_batch(local)[0], batch),
            "bfs_multi": lambda: all(np.array_equal(r, bfs[int(v)]) for r, v in zip(g.bfs_multi(srcs)[0], srcs)),
            "sssp": lambda: np.array_equal(g.sssp(s)[0], sssp),
            "cc": lambda: np.array_equal(g.cc()[0], labels),
            "pagerank": lambda: np.abs(gd.pagerank(tolerance=0.0, iter_num=20)[0] - rank).sum() < 1e-6,
            "ppr": check_ppr,
        }


@pytest.fixture(scope="module")
def calls():
    return Calls().calls


@pytest.fixture(autouse=True)
def loop_test_off():
    yield
    _lib.lib.mg_selftest_loops(_lib.MG_LOOP_TEST_OFF)


NAMES = ["bfs", "bfs_pred", "bfs_roots", "bfs_batch", "bfs_multi", "sssp", "cc", "pagerank", "ppr"]


@pytest.mark.parametrize("name", NAMES)
def test_error_behind_the_launch_leaves_the_graph_usable(name, calls):
    # the kernel runs on while the call leaves: its barriers count for the next run on the graph
    for _ in range(3):
        assert calls[name]()
        _lib.lib.mg_selftest_loops(_lib.MG_LOOP_TEST_FAIL)
        with pytest.raises(MapGraphError) as e:
            calls[name]()
        assert e.value.status == _lib.MG_ERR_CUDA
        _lib.lib.mg_selftest_loops(_lib.MG_LOOP_TEST_OFF)
        assert calls[name]()
        for other in NAMES:
            assert calls[other](), other


@pytest.mark.parametrize("name", NAMES)
def test_barrier_wait_that_runs_out(name, calls):
    for _ in range(3):
        _lib.lib.mg_selftest_loops(_lib.MG_LOOP_TEST_WAITS)
        with pytest.raises(MapGraphError) as e:
            calls[name]()
        assert e.value.status == _lib.MG_ERR_TIMEOUT
        _lib.lib.mg_selftest_loops(_lib.MG_LOOP_TEST_OFF)
        for other in [name, *NAMES]:
            assert calls[other](), other


@pytest.mark.parametrize("name", NAMES)
def test_refused_launch_runs_level_by_level(name, calls):
    _lib.lib.mg_kernel_launches(1)
    assert calls[name]()
    one = _lib.lib.mg_kernel_launches(1)
    for _ in range(2):
        _lib.lib.mg_selftest_loops(_lib.MG_LOOP_TEST_REFUSE)
        assert calls[name]()
        # (CC: without its BFS as many launches, sampling rounds instead)
        assert _lib.lib.mg_kernel_launches(1) > one or name == "cc"
        _lib.lib.mg_selftest_loops(_lib.MG_LOOP_TEST_OFF)
        assert calls[name]()
        _lib.lib.mg_kernel_launches(1)


def test_call_behind_unfinished_work_does_not_hold_up_other_threads(calls):
    # thread A's call is queued on a stream whose host function waits until this thread's calls have returned
    torch = pytest.importorskip("torch")
    hg = HostGraph.rmat(11, 8, seed=3)
    g, ref = Graph(hg), oracle.bfs(hg.row_offsets, hg.column_indices, 1)
    assert np.array_equal(g.bfs(1)[0], ref)
    stream, release, released, out = torch.cuda.Stream(), threading.Event(), [], []

    @C.CFUNCTYPE(None, C.c_void_p)
    def wait(_):
        released.append(release.wait(20))

    launch = C.CDLL("libcudart.so.12").cudaLaunchHostFunc
    launch.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p]
    assert launch(stream.cuda_stream, C.cast(wait, C.c_void_p), None) == 0
    t = threading.Thread(target=lambda: out.append(g.bfs(1, stream=stream.cuda_stream)[0]))
    t.start()
    time.sleep(0.5)
    for name in NAMES:
        assert calls[name](), name
    assert not out
    release.set()
    t.join(30)
    assert released == [True] and np.array_equal(out[0], ref)
