"""Launches that give up (a barrier wait that ran out, more evicted vertices than a launch ranks): the level is redone by
the kernels of one phase each from the labels it started with, and the result stays the oracle's. A wait that runs out is
stood for by the host, which treats finished launches as given up: their output has then overwritten what it could."""
import numpy as np
import pytest

import gpu_heipa as H
import oracle as O
from helpers import to_oracle

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
