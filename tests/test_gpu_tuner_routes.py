"""GPU tests of which tunables the autotuner tries: those that the route taken
on the handle reads, and no others."""
import pytest

pytestmark = pytest.mark.gpu

BASE = 3             # timings of the settings at the start
BFS_DIV, CC_DIV, BF_DIV = 8, 8, 8   # candidates, one of them (or none) the setting at the start
PULL = ("heavy_deg", "heavy_mode", "pull_ctas_per_sm", "cta_expand", "grid_expand")


@pytest.mark.parametrize("app", ["pagerank", "spmv", "bp", "cc"])
def test_nothing_to_choose(pm, app):
    with pm.Graph.rmat(11, 8, symmetric=app == "cc") as g:
        if app == "spmv":
            g.gen_weights_unit()
        before = g.tunables()
        rep = g.tune(app)
        assert rep["trials"] == BASE and rep["best_ms"] == rep["default_ms"] > 0
        assert g.tunables() == before


def test_mix_of_value_applications(pm):
    with pm.Graph.rmat(11, 8) as g:
        g.gen_weights_unit()
        before = g.tunables()
        assert g.tune(["pagerank", "spmv", "bp"])["trials"] == BASE
        assert g.tunables() == before


def test_traversals_keep_the_pull_settings(pm):
    with pm.Graph.rmat(11, 8, symmetric=True) as g:
        g.gen_weights_int()
        before = g.tunables()
        rep = g.tune("bfs")
        # a sweep of the divisor, a second one when the first moved it
        assert rep["trials"] <= BASE + 2 * BFS_DIV
        assert all(g.get_tunable(k) == before[k] for k in PULL)
        rep = g.tune(["bfs", "cc", "bellman_ford"])
        if g.get_tunable("bf_dense") == 2 and g.get_tunable("bf_delta") == 0:  # still the one launch
            assert all(g.get_tunable(k) == before[k] for k in PULL)


def test_host_driven_routes_offer_their_settings(pm):
    with pm.Graph.rmat(11, 8) as g:
        g.set_tunable("pull_stage", 1)  # label propagation round by round
        rep = g.tune("cc")
        assert rep["trials"] >= BASE + CC_DIV - 1 + 4 + 5 + 6 - 3
    with pm.Graph.rmat(11, 8) as g:
        g.set_tunable("cuda_graphs", 0)
        assert g.tune("bfs")["trials"] >= BASE + BFS_DIV - 1 + 4 + 5 - 2

