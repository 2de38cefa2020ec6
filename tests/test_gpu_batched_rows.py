"""GPU tests of the batched calls over rows in order of degree: in-degrees on
the edges of the row kinds and pieces, ragged vertex counts, sources and seeds
without in-edges or out-edges, every width of the column and lane layouts."""
import numpy as np
import pytest

from test_gpu_sorted_pull import _graph

pytestmark = pytest.mark.gpu

DEGREES = [0, 1, 2, 3, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 500, 1023, 1024, 1025, 4500]


def _og(oracle, seed=1, transpose=False, n=5003):
    off, idx = _graph(n, DEGREES, seed, transpose)
    return oracle.Graph(n, off, idx)


def _picks(og, k):
    """k vertices: the first two without in-edges, one without out-edges, the hub, then spread ones."""
    indeg = np.bincount(og.idx, minlength=og.n)
    special = [*np.nonzero(indeg == 0)[0][:2], *np.nonzero(og.out_degree() == 0)[0][:1], int(np.argmax(indeg))]
    rest = np.random.RandomState(k).randint(0, og.n, k)
    return np.concatenate([special, rest]).astype(np.int32)[:k]


@pytest.mark.parametrize("k", [1, 7, 8, 9, 16, 17, 31, 32])
@pytest.mark.parametrize("heavy", [64, 1024])
def test_ppr_widths(pm, oracle, k, heavy):
    og = _og(oracle)
    seeds = _picks(og, k)
    with pm.Graph.from_csr(og.off, og.idx) as g:
        g.set_tunable("heavy_deg", heavy)
        for iters in (1, 2, 3, 6):
            want = oracle.ppr(og, seeds, iters)
            got = pm.PersonalizedPageRank(g, seeds, iters)
            # the suite's FP32 bound, per column
            assert (np.abs(got - want).sum(0) <= 1e-5 * np.abs(want).sum(0)).all(), iters
            assert np.array_equal(pm.PersonalizedPageRank(g, seeds, iters), got)


@pytest.mark.parametrize("k", [1, 2, 33, 64])
@pytest.mark.parametrize("transpose", [False, True])
def test_multi_source_traversals(pm, oracle, k, transpose):
    og = _og(oracle, 2, transpose)
    w = oracle.weights_int(og)
    sources = _picks(og, k)
    depth = np.stack([oracle.bfs(og, int(s))[0] for s in sources])
    dist = np.stack([oracle.dijkstra(og, w, int(s)) for s in sources])
    deg = og.out_degree()
    with pm.Graph.from_csr(og.off, og.idx, weights=w) as g:
        for thr in (-1, 0, 1 << 40, 70, og.m // 2):  # default, all dense, all sparse, switching
            got, st = pm.BFSMulti(sources, g, threshold=thr, stats=True)
            assert np.array_equal(got, depth), thr
            assert st["reached"] == (depth >= 0).sum() and st["edges_visited"] == ((depth >= 0) * deg).sum()
            assert np.array_equal(pm.BellmanFordMulti(sources, g, threshold=thr), dist), thr
        g.set_tunable("heavy_deg", 64)
        assert np.array_equal(pm.BellmanFordMulti(sources, g, threshold=0), dist)
