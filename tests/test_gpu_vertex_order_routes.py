"""GPU tests of the routes that pull and push in vertex order and of the
tunables they read (hub cache, heavy rows' cut-off and modes, staged ids, push
cut-offs): on a one-rank partition, which has no degree-sorted copy, on handles
whose copy found no memory, and on the host-driven rounds.  Launch counts show
that the route under test ran."""
import numpy as np
import pytest

from partition_local import LocalGroup

pytestmark = pytest.mark.gpu

RL1_F32 = 1e-5  # the suite's FP32 bound
ITERS = 6


def _rl1(a, b):
    return np.abs(np.asarray(a, np.float64) - b).sum() / np.abs(b).sum()


def _on_partition(pm, og, body, **kw):
    """body(handle) on the one-rank partition of og."""
    def run(rank, ex):
        with pm.Graph.partition(og.off, og.idx, rank, 1, ex, **kw) as g:
            return body(g)
    return LocalGroup(1).run(run)[0]


def _counted(pm, call):
    call()  # workspaces and tables
    pm.kernel_launches(reset=True)
    got = call()
    return got, pm.kernel_launches(reset=True)


@pytest.mark.parametrize("hub", [1, 100, 8192, 16384])
def test_hub_cache(pm, oracle, hub):
    og = oracle.rmat_graph(15, 16)

    def body(g):
        g.set_tunable("hub_cache", 0)
        base = _counted(pm, lambda: pm.PageRank(g, ITERS, dtype=np.float32))
        g.set_tunable("hub_cache", hub)
        return base, _counted(pm, lambda: pm.PageRank(g, ITERS, dtype=np.float32))

    (base, plain), (got, cached) = _on_partition(pm, og, body)
    assert np.array_equal(got, base)
    assert cached == plain + ITERS  # the cached sources' values, once a pass
    assert _rl1(base, oracle.pagerank(og, ITERS)) < RL1_F32


@pytest.mark.parametrize("heavy", [64, 1024, 1 << 30])
def test_heavy_rows(pm, oracle, heavy):
    og = oracle.rmat_graph(14, 16)
    w = oracle.weights_unit(og)
    x0 = oracle.uniform01(og.n)
    prior = oracle.uniform_open(2 * og.n).reshape(-1, 2)

    def body(g):
        g.set_tunable("heavy_deg", heavy)
        out = []
        for mode in (0, 1, 2):
            g.set_tunable("heavy_mode", mode)
            out.append([_counted(pm, lambda: pm.PageRank(g, ITERS)),
                        _counted(pm, lambda: pm.PageRank(g, ITERS, dtype=np.float32)),
                        _counted(pm, lambda: pm.SPMV(g, x0, ITERS)),
                        _counted(pm, lambda: pm.BeliefPropagation(g, prior, ITERS, dtype=np.float64))])
        return out

    runs = _on_partition(pm, og, body, weights=w)
    want = [oracle.pagerank(og, ITERS), oracle.pagerank(og, ITERS),
            oracle.spmv(og, w.astype(np.float64), x0.astype(np.float64), ITERS), oracle.bp(og, prior, ITERS)]
    split = heavy < np.diff(oracle_in_off(og)).max()
    for i, (tol, exact) in enumerate(((1e-10, None), (RL1_F32, None), (RL1_F32, None), (1e-10, None))):
        (m0, k0), (m1, k1), (m2, k2) = (runs[mode][i] for mode in (0, 1, 2))
        for got in (m0, m1, m2):
            assert _rl1(got, want[i]) < tol, (i, heavy)
        assert np.array_equal(m0, m2)  # the same chunks, folded in the same order
        if split:
            # a pass: chunks and pull; both in one launch; chunks beside the pull and a commit
            assert k0 - k1 == ITERS and k2 - k0 == ITERS, (i, k0, k1, k2)
        else:
            assert k0 == k1 == k2


def oracle_in_off(og):
    off = np.zeros(og.n + 1, np.int64)
    np.cumsum(np.bincount(og.idx, minlength=og.n), out=off[1:])
    return off


@pytest.mark.parametrize("scale", [10, 15])
def test_staged_ids(pm, oracle, scale):
    og = oracle.rmat_graph(scale, 16)
    prior = oracle.uniform_open(2 * og.n).reshape(-1, 2).astype(np.float32)

    def body(g):
        out = []
        for stage in (0, 1, 0, 1):
            g.set_tunable("pull_stage", stage)
            out.append([_counted(pm, lambda: pm.PageRank(g, ITERS, dtype=np.float32)),
                        _counted(pm, lambda: pm.PageRank(g, ITERS)),
                        _counted(pm, lambda: pm.BeliefPropagation(g, prior, ITERS))])
        return out

    runs = _on_partition(pm, og, body)
    assert _rl1(runs[1][0][0], oracle.pagerank(og, ITERS)) < RL1_F32
    for r in runs[1:]:
        for (a, ka), (b, kb) in zip(runs[0], r):
            assert np.array_equal(a, b) and ka == kb >= ITERS


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_whole_graph_without_memory_for_the_copy(pm, oracle, mode):
    og = oracle.rmat_graph(13, 16)
    want = oracle.pagerank(og, ITERS)
    with pm.Graph.from_csr(og.off, og.idx) as g:
        g.set_tunable("heavy_deg", 128)
        g.set_tunable("heavy_mode", mode)
        g.set_tunable("hub_cache", 512)
        for dtype, tol in ((np.float32, RL1_F32), (np.float64, 1e-10)):
            pm.PageRank(g, 0, dtype=dtype)  # staging
            pm.test_fail_alloc_after(1)
            try:
                pm.kernel_launches(reset=True)
                got = pm.PageRank(g, ITERS, dtype=dtype)
                launched = pm.kernel_launches(reset=True)
            finally:
                pm.test_fail_alloc_after(0)
            assert _rl1(got, want) < tol
            assert launched > 0


@pytest.mark.parametrize("cta,grid", [(32, 32), (32, 100000), (2048, 2048), (100000, 100000)])
def test_push_cut_offs(pm, oracle, cta, grid):
    sym = oracle.rmat_graph(13, 16, symmetric=True)
    w = oracle.weights_int(sym)
    srcs = oracle.pick_sources(sym, 2, seed=0x5EED0022)
    every = 1 << 40  # every round sparse
    with pm.Graph.from_csr(sym.off, sym.idx, symmetric=True, weights=w) as g:
        g.set_tunable("cta_expand", cta)
        g.set_tunable("grid_expand", grid)
        g.set_tunable("cuda_graphs", 0)  # BFS round by round
        g.set_tunable("cc_mode", 1)
        g.set_tunable("pull_stage", 1)   # Components round by round
        g.set_tunable("bf_dense", 0)     # BellmanFord round by round
        for s in srcs:
            pm.kernel_launches(reset=True)
            _, depth, st = pm.BFS(int(s), g, threshold=every, stats=True)
            assert pm.kernel_launches(reset=True) >= 2 * st["rounds"] and st["dense_rounds"] == 0
            assert np.array_equal(depth, oracle.bfs(sym, int(s))[0])
            dist, st = pm.BellmanFord(g, int(s), threshold=every, stats=True)
            assert pm.kernel_launches(reset=True) >= 2 * st["rounds"]
            assert np.array_equal(dist, oracle.dijkstra(sym, w, int(s)))
        labels, st = pm.Components(g, threshold=every, stats=True)
        assert pm.kernel_launches(reset=True) >= 2 * st["rounds"]
        assert np.array_equal(labels, oracle.cc(sym))


def test_bp_without_memory_for_the_counts(pm, oracle):
    og = oracle.rmat_graph(12, 8)
    prior = oracle.uniform_open(2 * og.n).reshape(-1, 2)
    with pm.Graph.from_csr(og.off, og.idx) as g, pm.Graph.from_csr(og.off, og.idx) as bare:
        g.set_tunable("cuda_graphs", 0)
        bare.set_tunable("cuda_graphs", 0)
        pm.BeliefPropagation(g, prior, 9, dtype=np.float64)
        pm.kernel_launches(reset=True)
        counts = pm.BeliefPropagation(g, prior, 9, dtype=np.float64)
        assert pm.kernel_launches(reset=True) == 1
        pm.BeliefPropagation(bare, prior, 0, dtype=np.float64)  # staging alone
        pm.test_fail_alloc_after(1)                             # the counts' first workspace
        try:
            pm.kernel_launches(reset=True)
            pulled = pm.BeliefPropagation(bare, prior, 9, dtype=np.float64)
            assert pm.kernel_launches(reset=True) >= 9
            with pm.Graph.from_csr(og.off, og.idx):  # the failure was met in that call
                pass
        finally:
            pm.test_fail_alloc_after(0)
    want = oracle.bp(og, prior, 9)
    for got in (counts, pulled):
        assert np.allclose(got, want, rtol=1e-9, atol=1e-12)  # the suite's FP64 bound
    assert np.allclose(counts, pulled, rtol=1e-12, atol=0)
