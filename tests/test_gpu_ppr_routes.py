"""GPU tests of personalised PageRank over the degree-sorted copy against the
vertex-order form (a handle without room for the copy) and the oracle: hubs of
several pieces, ragged slices, repeated seeds, replayed loops, no iterations."""
import numpy as np
import pytest

from test_gpu_batched_rows import _picks
from test_gpu_sorted_pull import _graph

pytestmark = pytest.mark.gpu

DEGREES = [9000, 2049, 2048, 2047, 1024, 1023, 129, 128, 127, 33, 32, 31, 5, 4, 3, 2, 1, 0]


@pytest.mark.parametrize("k", [1, 8, 9, 16, 17, 32])
def test_routes_agree(pm, oracle, k):
    for n in (9001, 9030, 33, 1):
        off, idx = _graph(n, DEGREES if n > 9000 else [], 7, False) if n > 1 else (np.zeros(2, np.int32), np.zeros(0, np.int32))
        og = oracle.Graph(n, off, idx)
        seeds = np.resize(_picks(og, 5) if n > 1 else [0], k).astype(np.int32)  # with repeats
        with pm.Graph.from_csr(off, idx) as g, pm.Graph.from_csr(off, idx) as bare:
            eye = np.zeros((n, k), np.float32)
            eye[seeds, np.arange(k)] = 1
            assert np.array_equal(pm.PersonalizedPageRank(bare, seeds, 0), eye)  # its workspaces
            for iters in (1, 2, 5):
                want = oracle.ppr(og, seeds, iters)
                first = pm.PersonalizedPageRank(g, seeds, iters)
                for _ in range(2):
                    assert np.array_equal(pm.PersonalizedPageRank(g, seeds, iters), first)
                pm.test_fail_alloc_after(1)  # the copy's first block
                try:
                    plain = pm.PersonalizedPageRank(bare, seeds, iters)
                finally:
                    pm.test_fail_alloc_after(0)
                for got in (first, plain):  # the suite's FP32 bound, per column
                    assert (np.abs(got - want).sum(0) <= 1e-5 * np.abs(want).sum(0)).all(), (n, iters)
