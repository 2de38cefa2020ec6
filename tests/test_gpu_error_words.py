"""GPU tests that an error word belongs to the call that met it: a later call on
the handle does not report it again."""
import ctypes as C
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

QUEUE_OVERFLOW, TIMEOUT = 1, 4  # DeviceError


@pytest.fixture(scope="module")
def words(pm):
    sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp"))
    import build
    L = C.CDLL(build.build("error_word"))
    L.leave_error_word.argtypes = [C.c_void_p, C.c_int, C.c_uint]
    L.read_error_words.argtypes = [C.c_void_p]
    return L


@pytest.mark.parametrize("slot,word", [(0, QUEUE_OVERFLOW), (0, TIMEOUT), (1, QUEUE_OVERFLOW), (2, TIMEOUT)])
def test_components_with_stats_after_a_failed_call(pm, oracle, words, slot, word):
    og = oracle.rmat_graph(10, 8, symmetric=True)
    with pm.Graph.from_csr(og.off, og.idx, symmetric=True) as g:
        assert words.leave_error_word(g.handle, slot, word) == 0
        labels, st = pm.Components(g, stats=True)
        assert np.array_equal(labels, oracle.cc(og))
        assert st["reached"] == og.n and st["rounds"] == 3 and st["edges_visited"] > 0


def test_an_error_is_reported_once(pm, oracle, words):
    og = oracle.rmat_graph(10, 8)
    with pm.Graph.from_csr(og.off, og.idx) as g:
        assert words.leave_error_word(g.handle, 1, TIMEOUT) == 0
        assert words.read_error_words(g.handle) == 4  # PM_ERR_TIMEOUT
        assert words.read_error_words(g.handle) == 0
