"""The single-launch coarsening level (one block, a cluster, a grid) against the oracle where it can go wrong: the
smallest graphs, the sizes at which the team changes, unit weights, rows around the lane / warp / block tiers, and leaf,
twin and relative groups from two members to most of the graph (ranked by counting or over a bitmap). The mapping is
compared directly, the coarse graphs through whole partitions. Integer results: equality."""
import numpy as np
import pytest

import gpu_heipa as H
import oracle as O
from helpers import isolated_plus_path, k2n, star, to_oracle

pytestmark = pytest.mark.gpu


def from_edges(n, edges, w=0):
    e = np.unique(np.sort(np.asarray(edges, np.int64), 1), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    both = np.concatenate([e, e[:, ::-1]])
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    xadj = np.concatenate([[0], np.cumsum(np.bincount(both[:, 0], minlength=n))])
    lo, hi = both.min(1), both.max(1)
    return H.Graph(xadj, both[:, 1], (lo * 7 + hi * 3) % w + 1 if w else None)


def twin_groups(sizes, w):
    """Groups of twins: the members of group i are adjacent to the hubs 2i and 2i + 1 only."""
    edges, v = [], 2 * len(sizes)
    for i, s in enumerate(sizes):
        for _ in range(s):
            edges += [(v, 2 * i), (v, 2 * i + 1)]
            v += 1
    return from_edges(v, edges, w)


def leaves_of(hubs, per_hub):
    edges = [(i, (i + 1) % hubs) for i in range(hubs)]
    v = hubs
    for h in range(hubs):
        for _ in range(per_hub(h)):
            edges.append((h, v))
            v += 1
    return from_edges(v, edges, 5)


GRAPHS = {
    "two": from_edges(2, [(0, 1)]),
    "triangle": from_edges(3, [(0, 1), (1, 2), (0, 2)], 3),
    "isolated": isolated_plus_path(301, 7),
    "path1024": isolated_plus_path(0, 1024),
    "path1025": isolated_plus_path(1, 1024),
    "grid16384": H.Graph.grid(128, 128, 1, 9, seed=4),
    "grid16385": H.Graph.grid(145, 113),
    "star5000": star(5000),
    "twins": twin_groups([2, 3, 31, 63, 64, 65, 66, 500], 7),
    "twins_unit": twin_groups([2, 3, 64, 65, 1500], 0),
    "k2n": k2n(20000),
    "leaves": leaves_of(61, lambda h: h + 3),
    "hub_rows": from_edges(2300, [(h, j) for h, ln in enumerate([31, 32, 33, 257, 1023, 1024, 1025, 2200])
                                  for j in range(50, 50 + ln)] + [(j, j + 1) for j in range(50, 2250)], 9),
    "rmat13": H.Graph.rmat(13, 8, seed=3),
    "rmat15": H.Graph.rmat(15, 12, seed=5),
    "rgg": H.Graph.rgg3d(40000, 9.0, 1, 50, seed=2),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_team_matching_and_contraction_equal_oracle(name):
    g = GRAPHS[name]
    og = to_oracle(g)
    c = H.Context(0, 1 << 30)
    try:
        dg = c.upload(g)
        mp, nc = c.match(dg)
        omp, onc = O.match(og)
        assert nc == onc
        np.testing.assert_array_equal(mp, omp)
        dg.free()
        part, cut = c.partition(g, 3, 0.03, "default", 5)
        want, want_cut = O.partition(og, 3, 0.03, False, 5)
        assert cut == want_cut
        np.testing.assert_array_equal(part, want)
    finally:
        c.close()


def test_long_coarse_rows_take_the_contraction_kernels():
    # a hub of 12000 entries: its coarse row exceeds the tables of every team
    g = H.Graph.rmat(14, 4, seed=9)
    e = [(0, j) for j in range(1, 12001)]
    rows = np.repeat(np.arange(g.n), np.diff(g.xadj.astype(np.int64)))
    g = from_edges(g.n, np.concatenate([np.stack([rows, g.adj.astype(np.int64)], 1), e]), 9)
    with H.Context(0, 1 << 30) as c:
        part, cut = c.partition(g, 8, 0.03, "default", 5)
    want, want_cut = O.partition(to_oracle(g), 8, 0.03, False, 5)
    assert cut == want_cut
    np.testing.assert_array_equal(part, want)


def wrapped_coarse_graph(n, deg, seed):
    """A graph and the mapping that pairs its vertices: the 1 to 4 entries between two pairs weigh up to 2^30 each, so
    coarse weights are sums below and above 2^31, 2^31 itself and 0 modulo 2^32."""
    rng = np.random.default_rng(seed)
    ring = [rng.permutation(n) for _ in range(deg // 2)]  # all degrees on one side of 16: neighbours see an edge alike
    a = np.concatenate([np.stack([p, np.roll(p, 1)], 1) for p in ring])
    e = np.concatenate([2 * a + np.array(x) for x in ((0, 0), (0, 1), (1, 0), (1, 1))])
    e = e[rng.random(len(e)) < 0.8]
    g = from_edges(2 * n, e, 1)
    rows = np.repeat(np.arange(g.n), np.diff(g.xadj.astype(np.int64)))
    key = np.minimum(rows, g.adj) + np.maximum(rows, g.adj)
    g.ew = np.array([1 << 30, 1 << 30, (1 << 29) + 1, 5, 1 << 30], np.int32)[key % 5]
    return g, (np.arange(g.n) // 2).astype(np.uint32)


@pytest.mark.parametrize("n,deg", [(700, 6), (700, 30), (9000, 12), (40000, 6), (40000, 26), (3000, 90)])
def test_matching_of_weights_that_wrapped(n, deg):
    g, mp = wrapped_coarse_graph(n, deg, n + deg)
    out = []
    for max_n in (1 << 20, 0):  # one launch, a launch per phase
        with H.Context(0, 512 << 20) as c:
            c.tune("match_coop_max_n", max_n)
            dg = c.upload(g)
            cg = c.contract(dg, mp, n)
            assert (cg.download().ew < 0).any() and (cg.download().ew == 0).any()
            out.append(c.match(cg))
    assert out[0][1] == out[1][1]
    np.testing.assert_array_equal(out[0][0], out[1][0])
