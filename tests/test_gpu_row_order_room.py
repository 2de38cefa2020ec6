"""GPU tests of the calls that take rows by in-degree on a handle without memory
for that order: they take them in vertex order, with the same results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _calls(pm, oracle, og, w):
    srcs = oracle.pick_sources(og, 20)
    depth = np.stack([oracle.bfs(og, int(s))[0] for s in srcs])
    dist = np.stack([oracle.dijkstra(og, w, int(s)) for s in srcs])
    ranks = oracle.ppr(og, srcs, 4)

    def bfs(g):
        assert np.array_equal(pm.BFSMulti(srcs, g, threshold=0), depth)

    def bf(g):
        assert np.array_equal(pm.BellmanFordMulti(srcs, g, threshold=0), dist)

    def ppr(g):
        got = pm.PersonalizedPageRank(g, srcs, 4)
        assert (np.abs(got - ranks).sum(0) <= 1e-5 * np.abs(ranks).sum(0)).all()

    return {"bfs": bfs, "bf": bf, "ppr": ppr}


@pytest.mark.parametrize("name", ["bfs", "bf", "ppr"])
def test_vertex_order(pm, oracle, name):
    og = oracle.rmat_graph(12, 16, symmetric=True)  # hubs, and vertices without edges
    w = oracle.weights_int(og)
    call = _calls(pm, oracle, og, w)[name]
    went_on = []
    for k in range(1, 24):
        with pm.Graph.from_csr(og.off, og.idx, symmetric=True, weights=w) as g:
            pm.test_fail_alloc_after(k)
            try:
                try:
                    call(g)
                    ok = True
                except pm.PolymerError as exc:  # a workspace the call cannot do without
                    assert exc.status == 2
                    ok = False
                # whether the failure was met: if not, the next allocations would meet it
                met = True
                try:
                    for _ in range(k):
                        pm.Graph.from_csr(np.zeros(3, np.int32), np.zeros(0, np.int32)).close()
                except pm.PolymerError:
                    met = False
            finally:
                pm.test_fail_alloc_after(0)
            if not met:
                break
            if ok:
                went_on.append(k)
            call(g)  # the handle is usable, with the order this time
    # the order's five arrays and the sort's own space, at least; a first failure that the call
    # went on from may belong to the sorted copy of PPR, which builds the order, too
    assert len(went_on) >= 5, went_on


def test_multi_source_bfs_with_little_memory(pm):
    """Three level slots and every row in vertex order: what is left when neither
    the sixteen slots (134 MB) nor the order's arrays (21 MB while it is built) fit."""
    import torch
    from test_gpu_reclaim import MB, Hog
    out = torch.empty((2, 1 << 20), dtype=torch.int32, device="cuda")
    with pm.Graph.rmat(20, 16, symmetric=True) as g, pm.Graph.rmat(20, 16, symmetric=True) as tight:
        srcs = np.array([1, 77], np.int32)
        want, st = pm.BFSMulti(srcs, g, stats=True)
        with Hog(pm, 64 * MB):
            for threshold in (0, -1, 1 << 40):
                got, st2 = pm.BFSMulti(srcs, tight, threshold=threshold, stats=True, out=out)
                assert np.array_equal(got.cpu().numpy(), want) and st2["reached"] == st["reached"]
