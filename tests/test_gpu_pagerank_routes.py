"""GPU tests of what PageRank's rules on the route leave to the vertex-order
form (a damping outside [0, 1]) and of replayed passes whose residual
workspace has moved since they were captured."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sign_rule(off, idx, iters, damping):
    """PageRank with the frontier in the contribution's sign, in FP64."""
    n = len(off) - 1
    deg = np.diff(off)
    src = np.repeat(np.arange(n), deg)
    p, q = np.full(n, 1.0 / n), np.zeros(n)
    share = np.where(deg > 0, 1.0 / n / np.maximum(deg, 1), 0.0)
    for _ in range(iters):
        acc = np.full(n, -0.0)
        np.add.at(acc, idx, share[src])
        in_f, hit = ~np.signbit(share), ~np.signbit(acc)
        q = np.where(in_f, damping * (q + acc) + (1.0 - damping) / n, q + acc)
        p = np.where(in_f, 0.0, p)
        share = np.where(hit, np.where(deg > 0, q / np.maximum(deg, 1), 0.0), -0.0)
        p, q = q, p
    return p


# with these values no sum of 1 / degree makes a rank exactly 0
@pytest.mark.parametrize("damping", [0.0, 0.85, 1.0, 1.27, -0.27])
def test_damping(pm, damping):
    rng = np.random.RandomState(11)
    n = 300
    pairs = np.unique(rng.randint(0, n, (900, 2)), axis=0)
    pairs = pairs[pairs[:, 0] != pairs[:, 1]]
    off = np.concatenate([[0], np.cumsum(np.bincount(pairs[:, 0], minlength=n))]).astype(np.int32)
    idx = pairs[:, 1].astype(np.int32)
    with pm.Graph.from_csr(off, idx) as g:
        g.set_parts([0, n])
        for iters in (1, 2, 5, 6):
            want = _sign_rule(off, idx, iters, damping)
            bound = np.abs(want).sum()
            assert np.abs(pm.PageRank(g, iters, damping) - want).sum() <= 1e-10 * bound
            # the suite's FP32 bound
            assert np.abs(pm.PageRank(g, iters, damping, dtype=np.float32) - want).sum() <= 1e-5 * bound
            assert np.abs(pm.PageRankParts(g, iters, damping) - want).sum() <= 1e-5 * bound


def test_replay_after_the_residual_workspace_moved(pm, oracle):
    og = oracle.rmat_graph(17, 4)
    w = oracle.weights_unit(og)
    with pm.Graph.from_csr(og.off, og.idx, weights=w) as g:
        g.set_parts([0, og.n])
        calls = [lambda: pm.PageRank(g, 4, resid=True), lambda: pm.SPMV(g, np.ones(og.n), 3, norms=True)]
        first = [c() for c in calls]
        for c in calls:  # captured, then replayed
            c(), c()
        pm.PageRankParts(g, 1)  # needs more of the same workspace
        for c, want in zip(calls, first):
            got = c()
            assert np.array_equal(got[0], want[0])
            assert np.allclose(got[1], want[1], rtol=1e-12, atol=0)
