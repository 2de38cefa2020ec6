"""GPU tests of fixed points with infinite values: a vertex without edges whose
value is infinite has no defined change (inf - inf), so the iteration runs to its
limit, and the other vertices still reach their values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 60


@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_adjoint_with_an_infinite_gradient(pm, oracle, value):
    og = oracle.rmat_graph(9, 8)
    n = og.n + 1  # the last vertex has no edges
    off = np.append(og.off, og.off[-1]).astype(np.int32)
    deg = np.diff(off)
    w = (np.ones(off[-1]) / np.repeat(deg, deg)).astype(np.float32)
    p = np.full(n, 1 / n, np.float32)
    grad = oracle.uniform01(n).astype(np.float32)
    with pm.Graph.from_csr(off, og.idx, weights=w) as g:
        _, want, _ = pm.PageRankAdjoint(g, p, grad, 0.85, 0.0, max_iters=LIMIT, with_lambda=True)
        grad[n - 1] = value
        _, lam, iters = pm.PageRankAdjoint(g, p, grad, 0.85, 1e-6, max_iters=LIMIT, with_lambda=True)
    assert iters == LIMIT
    assert lam[n - 1] == value and np.array_equal(lam[:-1], want[:-1])


def test_weighted_pagerank_of_an_edgeless_graph(pm):
    with pm.Graph.from_csr(np.zeros(34, np.int32), np.zeros(0, np.int32), weights=np.zeros(0, np.float32)) as g:
        p, iters, resid = pm.WeightedPageRank(g, -np.inf, 1e-6, max_iters=LIMIT)
        assert iters == LIMIT and np.isnan(resid) and np.isinf(p).all()
        p, iters, resid = pm.WeightedPageRank(g, 0.85, 1e-6, max_iters=LIMIT)
        assert iters == 2 and resid == 0.0 and np.array_equal(p, np.full(33, p[0]))
