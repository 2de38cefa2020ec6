"""GPU tests of belief propagation by peeled counts (whole graphs) against the
FP64 oracle and against the pull of a one-rank partition, where the frontier
shrinks differently: never, at once, level by level past several batches of
kept counts, through a row long enough to be shared by the grid, with self
loops and parallel edges, and without memory for the counts."""
import numpy as np
import pytest

from partition_local import LocalGroup

pytestmark = pytest.mark.gpu


def _path(n):
    return n, np.arange(n - 1), np.arange(1, n)


def _star(n):  # vertex 0 reaches all the others, which form a cycle and a tail
    s = np.concatenate([np.zeros(n - 1, np.int64), np.arange(1, n // 2), [n // 2], np.arange(n // 2 + 1, n - 1)])
    d = np.concatenate([np.arange(1, n), np.arange(2, n // 2 + 1), [1], np.arange(n // 2 + 2, n)])
    return n, s, d


def _layers(n, rng):  # a random acyclic graph: edges from lower to higher ids
    a, b = rng.randint(0, n, 4 * n), rng.randint(0, n, 4 * n)
    keep = a != b
    return n, np.minimum(a, b)[keep], np.maximum(a, b)[keep]


def _loops(n, rng):  # self loops and parallel edges stay in the counts
    s = rng.randint(0, n, 3 * n)
    return n, np.concatenate([s, s[: n // 3], np.arange(0, n, 7)]), \
        np.concatenate([rng.randint(0, n, 3 * n), s[: n // 3], np.arange(0, n, 7)])


def _csr(n, s, d):
    order = np.lexsort((d, s))
    s, d = s[order], d[order]
    off = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(s, minlength=n), out=off[1:])
    return off, d.astype(np.int32)


GRAPHS = {
    "single": lambda r: (1, np.zeros(0, np.int64), np.zeros(0, np.int64)),
    "edgeless": lambda r: (1025, np.zeros(0, np.int64), np.zeros(0, np.int64)),
    "path": lambda r: _path(37),
    "star": lambda r: _star(9001),
    "layers": lambda r: _layers(3001, r),
    "loops": lambda r: _loops(2047, r),
}


@pytest.mark.parametrize("iters", [0, 1, 3, 4, 5, 9, 14])
@pytest.mark.parametrize("name", sorted(GRAPHS) + ["rmat"])
def test_counts_match_oracle_and_pull(pm, oracle, name, iters):
    rng = np.random.RandomState(7)
    if name == "rmat":
        og = oracle.rmat_graph(13, 8)
        off, idx, n = og.off, og.idx, og.n
    else:
        n, s, d = GRAPHS[name](rng)
        off, idx = _csr(n, s, d)
        og = oracle.Graph(n, off, idx)
    prior = rng.uniform(0.05, 0.95, (n, 2))
    want = oracle.bp(og, prior, iters)
    with pm.Graph.from_csr(off, idx) as g:
        got = pm.BeliefPropagation(g, prior, iters, dtype=np.float64)
        got32 = pm.BeliefPropagation(g, prior.astype(np.float32), iters)
        assert np.array_equal(pm.BeliefPropagation(g, prior, iters, dtype=np.float64), got)
        pm.test_fail_alloc_after(1)
        try:  # a handle without memory for the counts pulls (or has its workspaces already)
            again = pm.BeliefPropagation(g, prior, iters, dtype=np.float64)
        except pm.PolymerError as exc:
            assert exc.status == 2
            again = got
        finally:
            pm.test_fail_alloc_after(0)
    # the tolerances of the FP64 and FP32 results everywhere else in the suite
    assert np.allclose(got, want, rtol=1e-9, atol=1e-12) and np.allclose(again, want, rtol=1e-9, atol=1e-12)
    if iters and idx.size:
        assert np.abs(got32 - want).sum() <= 1e-5 * np.abs(want).sum()

    def body(rank, ex):
        with pm.Graph.partition(off, idx, rank, 1, ex) as g:
            return pm.BeliefPropagation(g, prior, iters, dtype=np.float64)

    pulled = LocalGroup(1).run(body)[0]
    assert np.allclose(got, pulled, rtol=1e-12, atol=0)
