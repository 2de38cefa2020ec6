"""GPU tests of multi-source BellmanFord's dense rounds over weights that its
untested additions may not take: negative ones and ones near 2^30 and 2^31."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INF = (1 << 30) - 1  # the distance of a vertex that is not reached


def _relax(n, src, dst, w, source):
    dist = np.full(n, INF, np.int64)
    dist[source] = 0
    while True:
        ok = dist[src] < INF
        new = dist.copy()
        np.minimum.at(new, dst[ok], dist[src[ok]] + w[ok])
        if np.array_equal(new, dist):
            return dist
        dist = new


@pytest.mark.parametrize("kind", ["small", "negative", "large", "edge", "both"])
@pytest.mark.parametrize("k", [1, 8, 9, 50, 64])
def test_weights(pm, kind, k):
    rng = np.random.RandomState(3)
    n = 700
    pairs = np.unique(np.sort(rng.randint(0, n, (6000, 2)), axis=1), axis=0)  # edges go up: no cycles
    hub = np.stack([np.arange(n - 1), np.full(n - 1, n - 1)], 1)  # and all reach the last vertex
    pairs = np.unique(np.concatenate([pairs[pairs[:, 0] < pairs[:, 1]], hub]), axis=0)
    src, dst = pairs[:, 0], pairs[:, 1]
    w = rng.randint(1, 23, len(src))
    some = rng.uniform(size=len(src)) < 0.3
    if kind in ("negative", "both"):
        w[some] -= 25
    large = {"large": [0, 0, (1 << 30) + 100, (1 << 31) - 5000],  # from finite distances far below
             "edge": [0, 0, (1 << 30) - 30, 1 << 30], "both": [0, 0, (1 << 30) - 30, 1 << 30]}
    if kind in large:  # no sum of a finite distance and a weight passes 2^31
        pick = rng.choice(large[kind], len(src))
        w = np.where(~some & (pick > 0), pick, w)
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    sources = rng.randint(0, n // 4, k).astype(np.int32)
    # distances at or above INF are not paths the 32-bit distances can hold
    want = np.stack([np.minimum(_relax(n, src, dst, w, s), INF) for s in sources])
    with pm.Graph.from_csr(off, dst.astype(np.int32), weights=w.astype(np.int32)) as g:
        for thr in (-1, 0, 1 << 40):  # default, all dense, all sparse
            assert np.array_equal(pm.BellmanFordMulti(sources, g, threshold=thr), want), thr
