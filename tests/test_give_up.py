"""Launches that give up (a barrier wait that ran out, more evicted vertices than a launch ranks): the level is redone by
the kernels of one phase each from the labels it started with, and the result stays the oracle's. A wait that runs out is
stood for by the host, which treats finished launches as given up: their output has then overwritten what it could."""
import numpy as np
import pytest

import gpu_heipa as H
import oracle as O
from helpers import to_oracle
from test_jet_team import TEAMS, alternating

pytestmark = pytest.mark.gpu

RMAT = H.Graph.rmat(13, 8, seed=3)
MESH = H.Graph.rgg3d(30000, 9.0, 1, 50, seed=2)


def solve(g, k, config, **tunes):
    """(labels, cut, names of the timed launches)"""
    with H.Context(0, 1 << 30) as c:
        c.tune("jet_graph_max_m", 0)  # launches inside captured graphs have no timers
        for name, v in tunes.items():
            c.tune(name, v)
        c.instrument(True)
        part, cut = c.partition(g, k, 0.03, config, 5)
        names = [r[0] for r in c.kernel_log()]
    return part, cut, names


def count(names, prefix):
    return sum(n.startswith(prefix) for n in names)


@pytest.mark.parametrize("g", [RMAT, MESH], ids=["rmat", "mesh"])
def test_coarsening_launch_that_gives_up_is_made_once(g):
    want = O.partition(to_oracle(g), 6, 0.03, False, 5)
    _, _, plain = solve(g, 6, "default")
    part, cut, names = solve(g, 6, "default", team_give_up=1)
    assert cut == want[1]
    np.testing.assert_array_equal(part, want[0])
    assert count(names, "k_coarsen_team") == count(plain, "k_coarsen_team") > 0


GIVE_UP = {"wait": {"team_give_up": 2}, "evictions": {"jet_rank_pairs": 0}}
LOOP = ("k_lp_dispatch", "k_weak_pick", "k_strong_pick")  # passes of the per-kernel loop


@pytest.mark.parametrize("why", sorted(GIVE_UP))
@pytest.mark.parametrize("team", ["cluster", "grid"])
@pytest.mark.parametrize("config", ["default", "ultra"])
def test_levels_that_are_redone_in_a_partition(config, team, why):
    # the start labels are projected again
    tunes = dict(TEAMS["cluster"]) if team == "cluster" else {"jet_fused_max_n": 0}
    for g, k in ((RMAT, 48), (MESH, 300)):
        want = O.partition(to_oracle(g), k, 0.03, config == "ultra", 5)
        part, cut, names = solve(g, k, config, **tunes, **GIVE_UP[why])
        assert cut == want[1]
        np.testing.assert_array_equal(part, want[0])
        assert count(names, "k_jet") > 0 and count(names, LOOP) > 0


@pytest.mark.parametrize("config", ["IM", "HM"])
def test_levels_that_are_redone_in_a_mapping(config):
    hier, dist = [2, 4, 3], [1, 10, 100]
    og = to_oracle(MESH)
    want = O.map_im(og, hier, dist, 0.03, 5) if config == "IM" else O.map_hm(og, hier, dist, 0.03, False, 5)
    with H.Context(0, 1 << 30) as c:
        c.tune("team_give_up", 3)
        part, J = c.process_map(MESH, hier, dist, 0.03, config, 5)
    assert J == want[1]
    np.testing.assert_array_equal(part, want[0])


@pytest.mark.parametrize("why", sorted(GIVE_UP))
@pytest.mark.parametrize("team", ["cluster", "grid"])
def test_level_that_is_redone_in_a_refinement(team, why):
    # the start labels are those of the caller, over which the launch has written better ones before it gives up
    g, k = H.Graph.grid(200, 120, 1, 9, seed=2), 4
    part, lmax = alternating(g.n, k, 600)
    cut, maxw = O.edge_cut(to_oracle(g), part), int(np.bincount(part).max())
    want = O.jet_refine(to_oracle(g), k, lmax, False, 0, part, cut, maxw)
    with H.Context(0, 256 << 20) as c:
        c.tune("jet_graph_max_m", 0)
        for name, v in GIVE_UP[why].items():
            c.tune(name, v)
        for name, v in TEAMS[team].items():
            c.tune(name, v)
        dg = c.upload(g)
        c.instrument(True)
        got = c.jet_refine(dg, k, lmax, part, cut, maxw)
        names = [r[0] for r in c.kernel_log()]
    assert got[1:] == want[1:]
    np.testing.assert_array_equal(got[0], want[0])
    assert count(names, "k_jet") == 1 and count(names, LOOP) > 0
