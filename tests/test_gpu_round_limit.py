"""GPU tests of traversals that take more rounds than one launch runs: they go
on in further launches, from queues and from bitmaps, with the same results;
a negative cycle is given up after bounded launches, too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROUNDS = 1024  # kRoundsPerLaunch


def _path(n, both=True):
    s = np.concatenate([np.arange(n - 1), np.arange(1, n)] if both else [np.arange(n - 1)])
    d = np.concatenate([np.arange(1, n), np.arange(n - 1)] if both else [np.arange(1, n)])
    order = np.lexsort((d, s))
    off = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(s, minlength=n), out=off[1:])
    return off, d[order].astype(np.int32)


def _launches(pm, call):
    pm.kernel_launches(reset=True)
    got = call()
    return got, pm.kernel_launches(reset=True)


@pytest.mark.parametrize("n", [ROUNDS - 1, ROUNDS, ROUNDS + 1, ROUNDS + 2, 2 * ROUNDS + 1, 3 * ROUNDS + 7])
@pytest.mark.parametrize("threshold", [0, 4, 1 << 40])  # every round dense; from two frontier vertices on; sparse
def test_paths(pm, n, threshold):
    off, idx = _path(n)
    v = np.arange(n)
    mid = n // 2
    least = (n - 1) // ROUNDS  # launches beyond the first: a round per vertex of the path from its end
    with pm.Graph.from_csr(off, idx, symmetric=True, weights=np.full(idx.size, 3, np.int32)) as g:
        for s in (0, mid):
            (parents, depth, st), k = _launches(pm, lambda: pm.BFS(s, g, threshold=threshold, stats=True))
            assert np.array_equal(depth, abs(v - s)) and st["reached"] == n
            assert np.array_equal(parents[v != s], (v - np.sign(v - s))[v != s])
            dist, kd = _launches(pm, lambda: pm.BellmanFord(g, s, threshold=threshold))
            assert np.array_equal(dist, 3 * abs(v - s))
            if s == 0:
                assert k > least and kd > least
        sources = [0, n - 1, mid, mid]
        (many, st), k = _launches(pm, lambda: pm.BFSMulti(sources, g, threshold=threshold, stats=True))
        assert np.array_equal(many, [abs(v - s) for s in sources]) and st["reached"] == 4 * n
        assert k > least
        g.set_tunable("cc_mode", 1)
        labels, k = _launches(pm, lambda: pm.Components(g, threshold=threshold))
        assert not labels.any()


def test_labels_of_a_directed_path(pm, oracle):
    off, idx = _path(2 * ROUNDS + 5, both=False)
    og = oracle.Graph(2 * ROUNDS + 5, off, idx)
    with pm.Graph.from_csr(off, idx) as g:
        assert np.array_equal(pm.Components(g), oracle.cc(og))


def test_negative_cycle_comes_back(pm):
    n = 4 * ROUNDS
    off, idx = _path(n)
    with pm.Graph.from_csr(off, idx, symmetric=True, weights=np.full(idx.size, -1, np.int32)) as g:
        pm.kernel_launches(reset=True)
        with pytest.raises(pm.PolymerError) as ei:
            pm.BellmanFord(g, 0)
        assert "did not converge" in str(ei.value)
        assert pm.kernel_launches(reset=True) >= n // ROUNDS
        g.set_weights(np.full(idx.size, 2, np.int32))
        assert np.array_equal(pm.BellmanFord(g, 0), 2 * np.arange(n))
