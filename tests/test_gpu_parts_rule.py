"""GPU tests of which form of PageRank on parts a union takes: the layout by
position where it is faster, vertex order for rows far longer than the rest and
for many more small parts than run at once.  The launches of the first call after the
parts were set show which (building the layout takes kernels of its own)."""
import numpy as np
import pytest

from test_gpu_parts_layout import _random, _star, _union

pytestmark = pytest.mark.gpu

FEW, MANY = 24, 60  # parts below and above the number that run at once (32 to 37)
EDGES = 131072   # mean edges of a part from which every union takes the layout
BUILD = 4        # kernels before the size of the layout is known
FILL = 1         # and the one that fills it


def _rows(longest):
    def edges(rng, n):  # 8 edges a vertex, the first row as long as asked
        s, d = rng.randint(0, n, 8 * n), rng.randint(0, n, 8 * n)
        return np.concatenate([s, rng.permutation(n)[:longest]]), np.concatenate([d, np.zeros(min(longest, n), np.int64)])
    return edges


@pytest.mark.parametrize("kind,sizes,build", [
    (_random, [500] * FEW, BUILD + FILL),
    (_random, [500] * MANY, 0),                           # a second wave of small parts
    (_random, np.geomspace(318, 6360, 50).astype(int), BUILD + FILL),  # the few large ones decide
    (_star, [4097, 3], BUILD),                            # slots that are mostly padding
    (_star, [33, 20, 10], BUILD + FILL),                  # ... but no more than a short part's slices
    (_rows(100), [EDGES // 8 + 500] * MANY, BUILD + FILL),  # waves of large parts
    (_rows(2000), [EDGES // 8 + 500] * MANY, BUILD),        # with a long row each
])
def test_route(pm, oracle, kind, sizes, build):
    off, idx, base = _union(np.array(sizes), kind, 5)
    with pm.Graph.from_csr(off, idx) as g:
        g.set_parts(base)
        pm.PageRank(g, 0, dtype=np.float32)  # staging
        pm.kernel_launches(reset=True)
        got = pm.PageRankParts(g, 6)
        assert pm.kernel_launches(reset=True) == build + 1
        assert np.array_equal(pm.PageRankParts(g, 6), got)
        assert pm.kernel_launches(reset=True) == 1  # the choice is kept with the parts
    og = oracle.Graph(len(off) - 1, off, idx)
    for a, b in list(zip(base[:-1], base[1:]))[:4]:
        want = oracle.pagerank(oracle.subgraph(og, int(a), int(b)), 6)
        assert np.abs(got[a:b] - want).sum() <= 1e-5 * np.abs(want).sum()
