"""GPU tests of PageRank on the parts of a disjoint union by position (slices
of 32 rows, longest first): part sizes around whole slices, parts without
edges, rows of very unequal length (which fall back to vertex order), few and
no iterations, parts set again; against the FP64 oracle part by part."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _union(sizes, edges_of, seed):
    rng = np.random.RandomState(seed)
    s, d, base = [], [], np.concatenate([[0], np.cumsum(sizes)])
    for i, n in enumerate(sizes):
        a, b = edges_of(rng, n)
        keep = a != b
        pairs = np.unique(np.stack([a[keep], b[keep]], 1), axis=0)
        s.append(pairs[:, 0] + base[i])
        d.append(pairs[:, 1] + base[i])
    s, d = np.concatenate(s), np.concatenate(d)
    order = np.lexsort((d, s))
    off = np.zeros(base[-1] + 1, np.int32)
    np.cumsum(np.bincount(s, minlength=base[-1]), out=off[1:])
    return off, d[order].astype(np.int32), base


def _random(rng, n):
    return rng.randint(0, n, 6 * n), rng.randint(0, n, 6 * n)


def _sparse(rng, n):  # half of the vertices without in-edges
    return rng.randint(0, n, n), rng.randint(0, max(1, n // 2), n)


def _star(rng, n):  # one row as long as the part
    return np.arange(n), np.zeros(n, np.int64)


def _none(rng, n):
    return np.zeros(0, np.int64), np.zeros(0, np.int64)


def _check(pm, oracle, g, off, idx, base, iters):
    got = pm.PageRankParts(g, iters)
    og = oracle.Graph(len(off) - 1, off, idx)
    for a, b in zip(base[:-1], base[1:]):
        want = oracle.pagerank(oracle.subgraph(og, int(a), int(b)), iters)
        # the suite's FP32 bound, per part
        assert np.abs(got[a:b] - want).sum() <= 1e-5 * np.abs(want).sum(), (iters, a, b)
    assert np.array_equal(pm.PageRankParts(g, iters), got)


@pytest.mark.parametrize("kind", [_random, _sparse, _star, _none])
def test_part_shapes(pm, oracle, kind):
    sizes = np.array([1, 2, 31, 32, 33, 64, 65, 500, 4097, 3])
    off, idx, base = _union(sizes, kind, 3)
    with pm.Graph.from_csr(off, idx) as g:
        g.set_parts(base)
        for iters in (0, 1, 2, 5, 6):
            _check(pm, oracle, g, off, idx, base, iters)


def test_hub_rows_and_parts_set_again(pm, oracle):
    og = oracle.rmat_graph(12, 8)
    n = og.n
    off = np.concatenate([og.off, og.off[-1] + og.off[1:]]).astype(np.int32)
    idx = np.concatenate([og.idx, og.idx + n]).astype(np.int32)
    with pm.Graph.from_csr(off, idx) as g:
        for base in ([0, n, 2 * n], [0, 2 * n], [0, n, 2 * n]):
            g.set_parts(base)
            got = pm.PageRankParts(g, 7)
            size = base[1]
            whole = oracle.Graph(size, off[:size + 1], idx[:off[size]])
            want = np.tile(oracle.pagerank(whole, 7), len(base) - 1)
            assert np.abs(got - want).sum() <= 1e-5 * np.abs(want).sum()
