"""GPU tests of Components by union-find on graphs of low degree: grids with and
without edges taken out (one component, one large and many small, many small),
long chains in id order and against it, rows on both sides of the length that a
lane links alone; labels exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(rng, h, w, drop):
    v = np.arange(h * w).reshape(h, w)
    s = np.concatenate([v[:, :-1].ravel(), v[:-1].ravel()])
    d = np.concatenate([v[:, 1:].ravel(), v[1:].ravel()])
    keep = rng.uniform(size=s.size) >= drop
    return h * w, s[keep], d[keep]


def _stars(rng, degrees):  # a hub each, its leaves elsewhere
    n = int(sum(degrees)) + len(degrees)
    v = rng.permutation(n)
    hubs, leaves = v[: len(degrees)], v[len(degrees):]
    return n, np.repeat(hubs, degrees), leaves


GRAPHS = {
    "grid": lambda r: _grid(r, 301, 203, 0.0),
    "grid without 3 in 10": lambda r: _grid(r, 512, 515, 0.3),
    "grid without half": lambda r: _grid(r, 400, 401, 0.5),
    "grid without 8 in 10": lambda r: _grid(r, 300, 301, 0.8),
    "path": lambda r: (70001, np.arange(70000), np.arange(1, 70001)),
    "path of every third, backwards": lambda r: (30000, np.arange(29999, 2, -1), np.arange(29996, -1, -1)),
    "shuffled path": lambda r: (lambda p: (20000, p[:-1], p[1:]))(r.permutation(20000)),
    "stars": lambda r: _stars(r, [15, 16, 17, 31, 32, 33, 100, 1, 2, 3] * 40),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_labels_exact(pm, oracle, name):
    n, s, d = GRAPHS[name](np.random.RandomState(11))
    og = oracle.graph_from_edges(n, s, d, symmetric=True)
    want = oracle.cc(og)
    with pm.Graph.from_csr(og.off, og.idx, symmetric=True) as g:
        for _ in range(3):
            assert np.array_equal(pm.Components(g), want)
