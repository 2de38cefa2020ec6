"""GPU tests of the pulls over the degree-sorted adjacency copy (PageRank,
SpMV, weighted PageRank, its adjoint, SpMV backward): rows whose degrees sit
on the edges of the row kinds and pieces, ragged vertex counts, rows without
edges, hubs of many pieces; against the FP64 oracle, and PageRank and SpMV
against the vertex-order pull of a one-rank partition."""
import numpy as np
import pytest

from partition_local import LocalGroup

pytestmark = pytest.mark.gpu

# below / at / above the cuts (32, 128), one and several pieces of 128 edges
DEGREES = [0, 1, 2, 3, 4, 5, 31, 32, 33, 63, 64, 127, 128, 129, 255, 256, 257, 384, 1023, 1025, 2999]


def _graph(n, degrees, seed, transpose):
    """n vertices whose in-degrees (out-degrees with transpose) run through
    `degrees`, then 0, 1, 2, ... cyclically up to 6; no self loops, no parallel edges."""
    rng = np.random.RandomState(seed)
    s, d = [], []
    for v in range(n):
        k = degrees[v] if v < len(degrees) else (v * 7) % 7
        k = min(k, n - 1)
        src = rng.choice(n - 1, k, replace=False)
        src[src >= v] += 1
        s.append(src)
        d.append(np.full(k, v))
    s, d = np.concatenate(s), np.concatenate(d)
    if transpose:
        s, d = d, s
    order = np.lexsort((d, s))
    s, d = s[order], d[order]
    off = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(s, minlength=n), out=off[1:])
    return off, d.astype(np.int32)


def _cases(oracle):
    yield "degrees", *_graph(3001, DEGREES, 1, False)
    yield "out-degrees", *_graph(3001, DEGREES, 2, True)
    yield "short", *_graph(67, [], 3, False)
    yield "single", np.zeros(2, np.int32), np.zeros(0, np.int32)
    yield "edgeless", np.zeros(34, np.int32), np.zeros(0, np.int32)
    og = oracle.rmat_graph(15, 16)
    yield "rmat", og.off, og.idx


def _rel(a, b):
    return np.abs(np.asarray(a, np.float64) - b).sum() / max(np.abs(b).sum(), 1e-300)


def test_against_oracle_and_vertex_order_pull(pm, oracle):
    for name, off, idx in _cases(oracle):
        og = oracle.Graph(len(off) - 1, off, idx)
        rng = np.random.RandomState(5)
        w = (1.0 - rng.uniform(size=og.m)).astype(np.float32)
        x0 = rng.uniform(size=og.n)
        with pm.Graph.from_csr(off, idx, weights=w) as g:
            for iters in (0, 1, 2, 3, 6, 7):
                want, resid = oracle.pagerank(og, iters, with_resid=True)
                got, r = pm.PageRank(g, iters, resid=True)
                # the suite's tolerances: FP64 1e-10 per element, FP32 1e-5 relative L1
                assert np.allclose(got, want, rtol=1e-10, atol=0), (name, iters)
                assert np.allclose(r, resid, rtol=1e-9, atol=1e-15), (name, iters)
                assert np.array_equal(pm.PageRank(g, iters), got), (name, iters)  # with and without residuals
                assert _rel(pm.PageRank(g, iters, dtype=np.float32), want) < 1e-5, (name, iters)
                y = oracle.spmv(og, w.astype(np.float64), x0, iters)
                got, norms = pm.SPMV(g, x0, iters, norms=True, dtype=np.float64)
                assert np.allclose(got, y, rtol=1e-10, atol=0), (name, iters)
                assert iters == 0 or np.isclose(norms[-1], np.abs(y).sum(), rtol=1e-10), (name, iters)
                assert _rel(pm.SPMV(g, x0.astype(np.float32), iters), y) < 1e-5 or not y.any(), (name, iters)

        def body(rank, ex):
            with pm.Graph.partition(off, idx, rank, 1, ex, weights=w) as p:
                return pm.PageRank(p, 6), pm.SPMV(p, x0, 3, dtype=np.float64)

        pr, sp = LocalGroup(1).run(body)[0]
        with pm.Graph.from_csr(off, idx, weights=w) as g:
            assert np.allclose(pm.PageRank(g, 6), pr, rtol=1e-12, atol=0), name
            assert np.allclose(pm.SPMV(g, x0, 3, dtype=np.float64), sp, rtol=1e-12, atol=0), name


@pytest.mark.parametrize("name", ["degrees", "out-degrees", "short", "single", "edgeless"])
def test_fixed_points_and_backward(pm, oracle, name):
    off, idx = {c[0]: c[1:] for c in _cases(oracle)}[name]
    og = oracle.Graph(len(off) - 1, off, idx)
    w = oracle.lognormal_weights(og).astype(np.float32)
    w64 = w.astype(np.float64)
    rng = np.random.RandomState(9)
    gp = rng.uniform(size=og.n).astype(np.float32)
    with pm.Graph.from_csr(off, idx, weights=w) as g:
        for tol, most in ((1e-6, 1000), (0.0, 3), (0.0, 17), (1e30, 5)):
            want, it = oracle.weighted_pagerank(og, w64, tol=tol, max_iters=most)
            p, got_it, res = pm.WeightedPageRank(g, tol=tol, max_iters=most)
            # the stopping pass may differ where the change lies at the tolerance, and FP32 may
            # reach its exact fixed point (no change at all, which meets tol = 0) before FP64 does
            assert got_it == it or (tol == 1e-6 and abs(got_it - it) <= 2) or (res == 0.0 and got_it < it)
            assert res <= tol or got_it == most
            assert _rel(p, want) < 5e-6
            dw_want, lam_want, it = oracle.pagerank_adjoint(og, w64, want, gp, tol=tol, max_iters=most)
            dw, lam, got_it = pm.PageRankAdjoint(g, want.astype(np.float32), gp, tol=tol, max_iters=most, with_lambda=True)
            assert got_it == it or (tol == 1e-6 and abs(got_it - it) <= 2) or (tol == 0.0 and got_it < it)
            assert _rel(lam, lam_want) < 5e-6 and (og.m == 0 or _rel(dw, dw_want) < 5e-6)
        g.profile(True)  # profiled passes are counted one by one
        _, n_it, _ = pm.WeightedPageRank(g, tol=1e-6)
        assert g.profile_read("weighted_pagerank", reset=True)[1] == n_it
        g.profile(False)
        x, gy = rng.uniform(size=og.n).astype(np.float32), rng.uniform(size=og.n).astype(np.float32)
        dx, dw = pm.SpMVBackward(g, x, gy)
        dx_want, dw_want = oracle.spmv_backward(og, w64, x.astype(np.float64), gy.astype(np.float64))
        assert og.m == 0 or _rel(dx, dx_want) < 1e-6 and _rel(dw, dw_want) < 1e-7
        assert og.m > 0 or not dx.any()
        g.set_weights(w * np.float32(0.5))  # new weights reach the copies
        assert og.m == 0 or np.allclose(pm.SpMVBackward(g, x, gy)[0], dx * 0.5, rtol=1e-6, atol=1e-30)
        assert _rel(pm.SPMV(g, x, 2), oracle.spmv(og, w64 * 0.5, x.astype(np.float64), 2)) < 1e-5 or og.m == 0
