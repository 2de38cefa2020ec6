"""GPU tests of label propagation's dense rounds, which pull: in-degrees on the
edges of the row kinds (a thread, eight lanes, a warp, a CTA per piece) and of
the pieces, rounds all dense, mixed and all sparse; labels exact against the
oracle, repeated calls alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEGREES = [40000, 32768, 16385, 16384, 16383, 1025, 1024, 1023, 129, 128, 127, 33, 32, 31, 5, 4, 3, 2, 1, 0]


def _graph(oracle, n, degrees, seed):
    """In-degrees run through `degrees` at random vertices, then 0 .. 3."""
    rng = np.random.RandomState(seed)
    deg = rng.randint(0, 4, n)
    deg[rng.permutation(n)[: len(degrees)]] = np.minimum(degrees, n - 1)
    d = np.repeat(np.arange(n), deg)
    s = rng.randint(0, n, d.size) if n < 100 else np.concatenate([rng.choice(n, k, replace=False) for k in deg])
    keep = s != d
    return oracle.graph_from_edges(n, s[keep], d[keep], symmetric=False)


@pytest.mark.parametrize("n,degrees", [(1, []), (33, []), (2049, DEGREES[5:]), (40001, DEGREES)])
def test_labels_exact(pm, oracle, n, degrees):
    og = _graph(oracle, n, degrees, n)
    want = oracle.cc(og)
    with pm.Graph.from_csr(og.off, og.idx) as g:
        for threshold in (0, max(1, len(og.idx) // 2), -1, 1 << 40):
            for _ in range(2):
                labels, st = pm.Components(g, threshold=threshold, stats=True)
                assert np.array_equal(labels, want)
            assert st["dense_rounds"] == (st["rounds"] if threshold == 0 else 0 if threshold == 1 << 40 else st["dense_rounds"])
