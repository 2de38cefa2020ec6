"""GPU tests of the arrays BFS takes for its results on the device: one array
for both (the depths are written last), arrays that overlap, addresses that are
not aligned to an element, either result alone."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def case(pm, oracle):
    og = oracle.rmat_graph(11, 8, symmetric=True)
    s = int(oracle.pick_sources(og, 1)[0])
    with pm.Graph.from_csr(og.off, og.idx, symmetric=True) as g:
        yield g, s, oracle.bfs(og, s)[0]


def _bfs(pm, g, s, parents, depth):
    pm._check(pm.lib().pm_bfs(g.handle, s, C.c_void_p(parents), C.c_void_p(depth), 1, -1, None))


def test_one_array_for_both(pm, case):
    import torch
    g, s, want = case
    buf = torch.zeros(g.n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    _bfs(pm, g, s, buf.data_ptr(), buf.data_ptr())
    assert np.array_equal(buf.cpu().numpy(), want)


def test_overlapping_arrays(pm, case):
    import torch
    g, s, want = case
    buf = torch.zeros(g.n + 7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    _bfs(pm, g, s, buf.data_ptr(), buf.data_ptr() + 28)
    assert np.array_equal(buf[7:].cpu().numpy(), want)


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_unaligned_arrays(pm, case, shift):
    import torch
    g, s, want = case
    p = torch.zeros(4 * g.n + 4, dtype=torch.uint8, device="cuda")
    d = torch.zeros(4 * g.n + 4, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    _bfs(pm, g, s, p.data_ptr() + shift, d.data_ptr() + shift)
    got = np.frombuffer(d.cpu().numpy().tobytes()[shift:shift + 4 * g.n], np.int32)
    parents = np.frombuffer(p.cpu().numpy().tobytes()[shift:shift + 4 * g.n], np.int32)
    assert np.array_equal(got, want)
    hit = (want > 0)
    assert np.array_equal(want[parents[hit]], want[hit] - 1) and parents[s] == s


def test_either_alone(pm, case):
    import torch
    g, s, want = case
    d = torch.zeros(g.n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    _bfs(pm, g, s, None, d.data_ptr())
    assert np.array_equal(d.cpu().numpy(), want)
    p = torch.zeros(g.n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    _bfs(pm, g, s, p.data_ptr(), None)
    got = p.cpu().numpy()
    assert got[s] == s and np.array_equal(want[got[want > 0]], want[want > 0] - 1)
