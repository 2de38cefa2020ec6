"""GPU tests of a handle that finds no room for its degree-sorted copy: the build
is not tried again, call after call, until the device has the memory."""
import numpy as np
import pytest

from test_gpu_reclaim import MB, SCALE, Hog

pytestmark = pytest.mark.gpu

ITERS = 6
VERTEX_ORDER = 1 + 2 * ITERS  # the start; heavy rows and pull, each pass


def _launches(pm, g):
    pm.kernel_launches(reset=True)
    ranks = pm.PageRank(g, ITERS, dtype=np.float32)
    return pm.kernel_launches(reset=True), ranks


def test_no_room(pm):
    with pm.Graph.rmat(SCALE, 16) as g:
        with Hog(pm, 200 * MB):  # a copy takes about 350 MB
            first, ranks = _launches(pm, g)
            assert first >= VERTEX_ORDER
            for _ in range(3):
                again, same = _launches(pm, g)
                assert again == VERTEX_ORDER and np.array_equal(same, ranks)
        _launches(pm, g)  # builds it
        after, same = _launches(pm, g)
        assert after < VERTEX_ORDER and np.abs(same - ranks).sum() < 1e-5


def test_a_copy_given_back_waits_for_its_room(pm):
    with pm.Graph.rmat(SCALE, 16) as g:
        _launches(pm, g)
        with_copy, ranks = _launches(pm, g)
        assert with_copy < VERTEX_ORDER
        with Hog(pm, 200 * MB):
            with pm.Graph.rmat(SCALE - 2, 16):  # takes the copy's memory, and goes on holding some
                counts = [_launches(pm, g)[0] for _ in range(3)]
        assert counts[1] == counts[2]  # no build in either
        _launches(pm, g)
        after, same = _launches(pm, g)
        assert after == with_copy and np.array_equal(same, ranks)
