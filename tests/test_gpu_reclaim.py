"""GPU tests of memory that handles hold only to make their calls faster (the
degree-sorted copies): a new graph, and a call on another handle, that run out of
memory get it back from handles that no call is using, in any thread."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCALE = 22  # 4 M vertices, 67 M edges: a copy of about 0.35 GB
MB = 1 << 20


class Hog:
    """All of the device's free memory but `leave` bytes."""

    def __init__(self, pm, leave):
        import torch
        torch.cuda.empty_cache()
        pm.release_memory_cache()
        free = torch.cuda.mem_get_info()[0]
        self.keep = torch.empty(free - leave, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch
        self.keep = None
        torch.cuda.empty_cache()


def _with_copies(pm):
    g = pm.Graph.rmat(SCALE, 16)
    ranks = pm.PageRank(g, 3, dtype=np.float32)
    assert np.array_equal(pm.PageRank(g, 3, dtype=np.float32), ranks)
    return g, ranks


def test_a_new_graph_gets_the_memory(pm, oracle):
    og = oracle.rmat_graph(20, 16)
    g, ranks = _with_copies(pm)
    with g:
        with Hog(pm, 300 * MB):  # the new graph needs about 500 MB while it is built
            with pm.Graph.from_csr(og.off, og.idx) as other:
                assert np.allclose(pm.PageRank(other, 3), oracle.pagerank(og, 3), rtol=1e-10, atol=0)
        assert np.array_equal(pm.PageRank(g, 3, dtype=np.float32), ranks)  # built again


def test_a_call_on_another_handle_gets_the_memory(pm, oracle):
    og = oracle.rmat_graph(18, 16, symmetric=True)
    w = oracle.weights_int(og)
    srcs = oracle.pick_sources(og, 64)
    g, ranks = _with_copies(pm)
    with g, pm.Graph.from_csr(og.off, og.idx, symmetric=True, weights=w) as other:
        with Hog(pm, 96 * MB):  # distances of 64 sources: 67 MB, twice
            dist = pm.BellmanFordMulti(srcs, other)
        assert np.array_equal(dist[0], oracle.dijkstra(og, w, int(srcs[0])))
        assert np.array_equal(pm.PageRank(g, 3, dtype=np.float32), ranks)


def test_threads_run_while_others_run_out(pm, oracle):
    """Calls on the holder in one thread, builds that need its memory in another:
    every result is right, and a build fails only with PM_ERR_OOM while the
    holder is in use."""
    og = oracle.rmat_graph(20, 16)
    want = oracle.pagerank(og, 2)
    g, ranks = _with_copies(pm)
    wrong, built = [], []
    stop = threading.Event()

    def caller():
        while not stop.is_set():
            if np.abs(pm.PageRank(g, 3, dtype=np.float32) - ranks).sum() > 1e-5:
                wrong.append("ranks")

    with g:
        with Hog(pm, 500 * MB):
            t = threading.Thread(target=caller)
            t.start()
            try:
                for _ in range(12):
                    try:
                        with pm.Graph.from_csr(og.off, og.idx) as other:
                            built.append(np.allclose(pm.PageRank(other, 2), want, rtol=1e-10, atol=0))
                    except pm.PolymerError as exc:
                        if exc.status != 2:
                            wrong.append(str(exc))
            finally:
                stop.set()
                t.join()
        assert not wrong and all(built)
        assert np.abs(pm.PageRank(g, 3, dtype=np.float32) - ranks).sum() <= 1e-5
