"""GPU tests of calls that run out of device memory while the handle holds its
degree-sorted copies: the copies go back and the call runs without them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3])
def test_out_of_memory_gives_the_copies_back(pm, oracle, k):
    og = oracle.rmat_graph(13, 16)
    w = oracle.weights_unit(og)
    s = int(oracle.pick_sources(og, 1)[0])
    x0 = oracle.uniform01(og.n)
    with pm.Graph.from_csr(og.off, og.idx, weights=w) as g:
        g.set_parts([0, og.n])
        for again in range(2):  # with replayed loops the second time
            for _ in range(3):
                ranks = pm.PageRank(g, 4)
            parts = pm.PageRankParts(g, 4)
            pm.SPMV(g, x0, 2)
            pm.test_fail_alloc_after(k)
            try:  # new workspaces (the first time round) that there is no room for
                wide = pm.PersonalizedPageRank(g, [s] * (8 if again else 2), 3)
                f64 = pm.SPMV(g, x0, 2, dtype=np.float64)
            finally:
                pm.test_fail_alloc_after(0)
            assert np.allclose(f64, oracle.spmv(og, w, x0, 2), rtol=1e-10, atol=0)
            assert np.array_equal(wide[:, 0], wide[:, 1])
            # the copies are built again
            assert np.array_equal(pm.PageRank(g, 4), ranks)
            assert np.array_equal(pm.PageRankParts(g, 4), parts)
