"""GPU tests of the traversals whose rounds run in one launch (BFS,
BellmanFord, label-propagation Components): out-degrees on the edges of the
queues' row and piece lengths, ragged vertex counts, rounds forced sparse,
dense and alternating, isolated sources; depths, distances and labels exact
against the oracle, BFS statistics equal to the host loop's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEGREES = [0, 1, 2, 30, 31, 32, 33, 63, 64, 65, 255, 256, 257, 511, 512, 513, 2900]


def _graph(oracle, n, degrees, seed, symmetric):
    """Out-degrees run through `degrees` (at random vertices), then 0 .. 3."""
    rng = np.random.RandomState(seed)
    deg = rng.randint(0, 4, n)
    at = rng.permutation(n)[: len(degrees)]
    deg[at] = np.minimum(degrees, n - 1)
    s = np.repeat(np.arange(n), deg)
    d = np.concatenate([rng.choice(n, k, replace=False) for k in deg]) if deg.sum() else np.zeros(0, np.int64)
    keep = s != d
    return oracle.graph_from_edges(n, s[keep], d[keep], symmetric=symmetric)


@pytest.mark.parametrize("n", [1, 31, 33, 3001])
@pytest.mark.parametrize("symmetric", [False, True])
def test_traversals_exact(pm, oracle, n, symmetric):
    og = _graph(oracle, n, DEGREES if n > 100 else [], n, symmetric)
    w = oracle.weights_int(og)
    labels = oracle.cc(og)
    rng = np.random.RandomState(3)
    sources = sorted({0, n - 1, int(np.argmax(og.out_degree())), *rng.randint(0, n, 3).tolist()})
    with pm.Graph.from_csr(og.off, og.idx, symmetric=symmetric, weights=w) as g:
        # every round sparse / every round dense / the default / switching in the middle
        for thr in (1 << 40, 0, -1, max(1, og.m // 3), max(1, og.m // 60), 70):
            g.set_tunable("cc_mode", 1)
            lab, st = pm.Components(g, threshold=thr, stats=True)
            assert np.array_equal(lab, labels), thr
            assert st["reached"] == n and st["dense_rounds"] <= st["rounds"]
            for s in sources:
                g.set_tunable("cuda_graphs", 1)
                par, depth, st = pm.BFS(s, g, threshold=thr, stats=True)
                assert np.array_equal(depth, oracle.bfs(og, s)[0]), (thr, s)
                assert np.array_equal(oracle.bfs_depths_from_parents(par, s), depth)
                for v in np.nonzero(depth > 0)[0][:50]:
                    row = og.idx[og.off[par[v]]:og.off[par[v] + 1]]
                    assert v in row
                g.set_tunable("cuda_graphs", 0)
                _, depth0, st0 = pm.BFS(s, g, threshold=thr, stats=True)
                assert np.array_equal(depth0, depth) and st0 == st, (thr, s)
                assert np.array_equal(pm.BellmanFord(g, s, threshold=thr), oracle.dijkstra(og, w, s)), (thr, s)


@pytest.mark.parametrize("n", [1, 2, 31, 2049, 60000])
def test_union_find_long_chains(pm, oracle, n):
    """Components by union-find where the trees are as deep as they get: a path
    in id order, in reverse, two interleaved, and rows in descending order."""
    for step in (1, 2):
        a = np.arange(n - step) if n > step else np.zeros(0, np.int64)
        og = oracle.graph_from_edges(n, a, a + step, symmetric=True)
        rows = [og.idx[og.off[v]:og.off[v + 1]][::-1] for v in range(n)]
        flipped = np.concatenate(rows) if n else og.idx
        for idx in (og.idx, flipped.astype(np.int32)):
            with pm.Graph.from_csr(og.off, idx, symmetric=True) as g:
                lab, st = pm.Components(g, stats=True)
                assert np.array_equal(lab, np.arange(n) % step if n > step else np.arange(n))
                assert st["edges_visited"] <= og.m


def test_profiled_rounds_are_counted(pm, oracle):
    og = oracle.rmat_graph(11, 8, symmetric=True)
    s = int(oracle.pick_sources(og, 1)[0])
    with pm.Graph.from_csr(og.off, og.idx, symmetric=True, weights=oracle.weights_int(og)) as g:
        g.profile(True)
        _, st = pm.BellmanFord(g, s, stats=True)
        ms, passes = g.profile_read("bellman_ford", reset=True)
        assert passes == st["rounds"] and ms > 0


def test_device_outputs_and_odd_alignment(pm, oracle):
    """Results written straight into CUDA buffers, also 4-byte aligned ones."""
    import torch
    og = oracle.rmat_graph(12, 8, symmetric=True)
    w = oracle.weights_int(og)
    s = int(oracle.pick_sources(og, 1)[0])
    n = og.n
    with pm.Graph.from_csr(og.off, og.idx, symmetric=True, weights=w) as g:
        g.set_tunable("cc_mode", 1)
        for shift in (0, 1, 3):
            buf = [torch.full((n + 4,), 77, dtype=torch.int32, device="cuda") for _ in range(4)]
            out = [b[shift:shift + n] for b in buf]
            pm.BFS(s, g, out=(out[0], out[1]))
            pm.BellmanFord(g, s, out=out[2])
            pm.Components(g, out=out[3])
            assert np.array_equal(out[1].cpu().numpy(), oracle.bfs(og, s)[0])
            assert np.array_equal(out[2].cpu().numpy(), oracle.dijkstra(og, w, s))
            assert np.array_equal(out[3].cpu().numpy(), oracle.cc(og))
            for b in buf:
                assert (b[:shift] == 77).all() and (b[shift + n:] == 77).all()
