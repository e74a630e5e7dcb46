"""The single-launch Jet level loop (block, cluster and cooperative-grid teams) against the oracle at the sizes where it
can go wrong: levels of one to a few vertices, row lengths around the tiers (8 lanes x 4 entries, a warp, 64-entry and
1024-entry limits), block counts around the table layouts (256 / 257, 1024), several mini-buckets per gain bucket, one
overloaded block, evictions that need fallback slots, and more of them than a tile of the ranking holds. Weights whose
sums wrap are compared with the per-kernel loop (the oracle's rules for connections of 0 or less differ). Integer results:
equality."""
import numpy as np
import pytest

import gpu_heipa as H
import oracle as O
from helpers import isolated_plus_path, star, to_oracle

pytestmark = pytest.mark.gpu

# block: levels that fit its shared memory run in one block, larger ones as a cluster
TEAMS = {"block": {"jet_fused_max_n": 65536, "jet_fused_max_m": 1 << 30, "jet_coop_max_n": 0},
         "cluster": {"jet_fused_max_n": 65536, "jet_fused_max_m": 1 << 30, "jet_coop_max_n": 0, "jet_block_max_n": 0},
         "grid": {"jet_fused_max_n": 0, "jet_coop_max_n": 1 << 24, "jet_coop_max_deg": 1 << 20, "jet_coop_rows": 64}}


def wheel(lens):
    """Hubs of the given row lengths over one shared ring of vertices."""
    n_ring = max(lens)
    edges = {(i, (i + 1) % n_ring) for i in range(n_ring)} if n_ring > 2 else set()
    for h, ln in enumerate(lens):
        edges |= {(j, n_ring + h) for j in range(ln)}
    e = np.array(sorted({(min(a, b), max(a, b)) for a, b in edges}), np.int64)
    both = np.concatenate([e, e[:, ::-1]])
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    n = n_ring + len(lens)
    xadj = np.concatenate([[0], np.cumsum(np.bincount(both[:, 0], minlength=n))])
    lo, hi = both.min(1), both.max(1)
    return H.Graph(xadj, both[:, 1], (lo * 7 + hi * 3) % 9 + 1)


def weighted(g, seed):
    return H.Graph(g.xadj, g.adj, g.ew, np.random.default_rng(seed).integers(1, 40, g.n).astype(np.int32))


CASES = {
    "one_vertex": (isolated_plus_path(1, 0), 4, None),
    "path": (isolated_plus_path(3, 30), 2, None),
    "tier_rows": (wheel([1, 8, 31, 32, 33, 63, 64, 65, 127, 128, 129]), 5, None),
    "hub_rows": (wheel([1023, 1024, 1025, 1500, 2100]), 64, None),
    "star": (star(3000), 3, None),
    "k256": (H.Graph.rmat(12, 12, seed=4), 256, None),
    "k257": (H.Graph.rmat(12, 12, seed=5), 257, None),
    "k1024": (weighted(H.Graph.rmat(13, 8, seed=6), 1), 1024, None),
    "sections": (weighted(H.Graph.rgg3d(30011, 9.0, 1, 9, seed=2), 3), 2, None),
    "heavy_vertices": (weighted(H.Graph.grid(61, 67, 1, 5, seed=3), 5), 24, None),
    "map256": (H.Graph.rgg3d(6007, 30.0, 1, 50, seed=7), 256, ([4, 8, 8], [1, 10, 100])),
    "map_hubs": (wheel([40, 64, 65, 1024, 1030, 1300]), 24, ([2, 4, 3], [1, 10, 100])),
}


@pytest.mark.parametrize("team", sorted(TEAMS))
@pytest.mark.parametrize("start", ["spread", "one_block"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_team_loop_equals_oracle(name, start, team):
    g, k, hd = CASES[name]
    og = to_oracle(g)
    rng = np.random.default_rng(11)
    part = rng.integers(0, k, g.n).astype(np.uint32)
    if start == "one_block":  # most of the weight in the last block
        part[rng.random(g.n) < 0.6] = k - 1
    vw = np.ones(g.n, np.int64) if g.vw is None else g.vw
    lmax = O.lmax(g.total_weight(), k, 0.03)
    maxw = int(np.bincount(part, weights=vw, minlength=k).max())
    hier, dist = hd if hd else (None, None)
    obj = O.comm_cost(og, part, hier, dist) if hd else O.edge_cut(og, part)
    c = H.Context(0, 512 << 20)
    try:
        for t, v in TEAMS[team].items():
            c.tune(t, v)
        dg = c.upload(g)
        for ultra in ((False,) if hd else (False, True)):
            got = c.jet_refine(dg, k, lmax, part, obj, maxw, ultra=ultra, level=0, hierarchy=hier, distance=dist)
            want = O.jet_refine(og, k, lmax, ultra, 0, part, obj, maxw, hier, dist)
            assert got[1:] == want[1:]
            np.testing.assert_array_equal(got[0], want[0])
        dg.free()
    finally:
        c.close()


LOOPS = dict(TEAMS, kernels={"jet_fused_max_n": 0, "jet_coop_max_n": 0})


@pytest.mark.parametrize("loop", sorted(LOOPS))
@pytest.mark.parametrize("lmax", [-2147483000, -2 ** 30, -1, 0])
def test_limits_that_no_block_can_meet(lmax, loop):
    # every block is overloaded by its whole weight or more; block weights of about 3000 less the first limit exceed 31
    # bits: the weight to evict is a 64-bit difference, the one in the bucket key (as in the reference) a 32-bit one
    g, k = weighted(H.Graph.grid(31, 29, 1, 5, seed=3), 7), 6
    og = to_oracle(g)
    part = np.random.default_rng(3).integers(0, k, g.n).astype(np.uint32)
    maxw = int(np.bincount(part, weights=g.vw, minlength=k).max())
    cut = O.edge_cut(og, part)
    want = O.jet_refine(og, k, lmax, False, 0, part, cut, maxw)
    with H.Context(0, 64 << 20) as c:
        for name, v in LOOPS[loop].items():
            c.tune(name, v)
        got = c.jet_refine(c.upload(g), k, lmax, part, cut, maxw)
    assert got[1:] == want[1:]
    np.testing.assert_array_equal(got[0], want[0])


def runs_of_four(n, seed):
    """Runs of four vertices, each vertex joined to its run and to all of six other runs. Entries between even runs weigh
    2^30, so that four of them add up to 0 modulo 2^32; inside an even run 100, elsewhere 1 to 5."""
    r = n // 4
    order = np.random.default_rng(seed).permutation(r)  # place of a run -> its id
    place = np.argsort(order)
    rows, cols, w = [], [], []
    for d in (0, 1, 2, 6):
        a, b = np.arange(r), order[(place + d) % r]
        for i in range(4):
            for j in range(4):
                if d == 0 and i >= j:
                    continue
                rows.append(4 * a + i)
                cols.append(4 * b + j)
                even = (a % 2 == 0) & (b % 2 == 0)
                w.append(np.where(even, 100 if d == 0 else 1 << 30, (a + b + i + j) % 5 + 1))
    rows, cols, w = (np.concatenate(x) for x in (rows, cols, w))
    rows, cols, w = np.concatenate([rows, cols]), np.concatenate([cols, rows]), np.concatenate([w, w])
    at = np.lexsort((cols, rows))
    xadj = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=4 * r))])
    return H.Graph(xadj, cols[at], w[at].astype(np.int32))


def refine_both(g, k, part, lmax, tunes, hd=None, ultra=False):
    """jet_refine by a team and by the per-kernel loop (which has no size limits): (labels, objective, weight) of each."""
    hier, dist = hd if hd else (None, None)
    maxw = int(np.bincount(part, weights=g.vw, minlength=k).max())
    out = []
    for t in (tunes, {"jet_fused_max_n": 0, "jet_coop_max_n": 0}):
        with H.Context(0, 256 << 20) as c:
            for name, v in t.items():
                c.tune(name, v)
            dg = c.upload(g)
            obj = c.comm_cost(dg, part, hier, dist) if hd else c.edge_cut(dg, part)
            out.append(c.jet_refine(dg, k, lmax, part, obj, maxw, ultra=ultra, hierarchy=hier, distance=dist))
            dg.free()
    return out


# team -> (vertices, blocks, settings): cluster and grid levels on few warps, so that the rows of a table meet more blocks
# with connection 0 than the table has slots
HASHED = {"block": (300, 257, TEAMS["block"]), "cluster": (40000, 1000, TEAMS["cluster"]),
          "grid": (24000, 1000, dict(TEAMS["grid"], jet_coop_rows=1 << 20))}


@pytest.mark.parametrize("team", sorted(HASHED))
@pytest.mark.parametrize("ultra", [False, True])
def test_hashed_tables_when_connections_are_zero(ultra, team):
    n, k, tunes = HASHED[team]
    g = runs_of_four(n, 5)
    part = (np.arange(n) // 4 % k).astype(np.uint32)
    got, want = refine_both(g, k, part, 2 * int(np.bincount(part).max()), tunes, ultra=ultra)
    assert got[1:] == want[1:]
    np.testing.assert_array_equal(got[0], want[0])
    assert (got[0] != part).any()


def circulant(n, reach, w):
    """A ring in which every vertex is joined to the `reach` next and previous ones; w: weight of each ring distance."""
    off = np.concatenate([np.arange(-reach, 0), np.arange(1, reach + 1)])
    cols = (np.arange(n)[:, None] + off[None, :]) % n
    at = np.argsort(cols, axis=1)
    ew = np.asarray(w, np.int64)[np.abs(off) - 1][at]
    return H.Graph(np.arange(n + 1) * 2 * reach, np.take_along_axis(cols, at, 1).ravel(), ew.ravel().astype(np.int32))


@pytest.mark.parametrize("team", ["block", "cluster", "grid"])
@pytest.mark.parametrize("k", [75, 300])
@pytest.mark.parametrize("reach", [9, 16, 20, 600])
def test_gains_at_the_ends_of_the_range(reach, k, team):
    # connections and gains of -2^31 (two entries of 2^30; a connection of 0 less one of -2^31) are values as all others
    n, k = (300, k // 4) if team == "block" else (6000, k)
    if 2 * reach >= n:
        pytest.skip("no such ring")
    g = circulant(n, reach, np.full(reach, 1 << 30))
    part = (np.arange(n) // 4 % k).astype(np.uint32)
    part[::37] = (part[::37] + 1) % k
    maxw = int(np.bincount(part).max())
    for lmax in (maxw, 2 * maxw):
        got, want = refine_both(g, k, part, lmax, TEAMS[team])
        assert got[1:] == want[1:]
        np.testing.assert_array_equal(got[0], want[0])


@pytest.mark.parametrize("team", ["block", "cluster", "grid"])
@pytest.mark.parametrize("kind", ["k40", "k300", "map"])
@pytest.mark.parametrize("reach", [2, 5, 8, 9])
def test_short_rows_with_blocks_of_connection_zero(reach, kind, team):
    # rows of up to 16 entries take a block whose weights add up to 0 for a neighbour, longer ones don't
    n = 300 if team == "block" else 6000
    k, hd = {"k40": (40, None), "k300": (300, None), "map": (24, ([2, 4, 3], [1, 10, 100]))}[kind]
    g = circulant(n, reach, np.full(reach, 1 << 30))
    part = (np.arange(n) * k // n).astype(np.uint32)
    part[::11] = part[::-11][:len(part[::11])]
    maxw = int(np.bincount(part, minlength=k).max())
    for lmax in (n // k + 1, maxw, 2 * maxw):
        got, want = refine_both(g, k, part, lmax, TEAMS[team], hd)
        assert got[1:] == want[1:]
        np.testing.assert_array_equal(got[0], want[0])


def alternating(n, k, over):
    """Blocks that are in turn larger and smaller than the average, and a limit `over` vertices in all below it: after two
    weak steps every second block is overloaded and strong rebalancing evicts about `over` vertices."""
    sizes = np.full(k, n // k)
    sizes[0::2] += n // k // 50
    sizes[1::2] -= n // k // 50
    return np.repeat(np.arange(k), sizes).astype(np.uint32), n // k - over // k


@pytest.mark.parametrize("team,tunes", [("cluster", TEAMS["cluster"]), ("grid", TEAMS["grid"]),
                                        ("two_blocks", dict(TEAMS["grid"], jet_coop_rows=1 << 20))])
@pytest.mark.parametrize("over", [120, 512, 516, 1020, 1024, 1032, 3000])
def test_ranks_of_evicted_vertices(over, team, tunes):
    # below, at and above a tile (512 or 1024 vertices), and several rounds of a warp's two vertices
    g, k = H.Graph.grid(200, 120), 4
    part, lmax = alternating(g.n, k, over)
    og = to_oracle(g)
    cut, maxw = O.edge_cut(og, part), int(np.bincount(part).max())
    want = O.jet_refine(og, k, lmax, False, 0, part, cut, maxw)
    with H.Context(0, 256 << 20) as c:
        for name, v in tunes.items():
            c.tune(name, v)
        got = c.jet_refine(c.upload(g), k, lmax, part, cut, maxw)
    assert got[1:] == want[1:]
    np.testing.assert_array_equal(got[0], want[0])


@pytest.mark.parametrize("kind", ["cut", "map"])
@pytest.mark.parametrize("tunes", [TEAMS["cluster"], dict(TEAMS["grid"], jet_coop_rows=1 << 20)], ids=["cluster", "grid"])
def test_more_long_rows_than_a_block_shares(tunes, kind):
    # 3000 rows of 300 entries in at most 16 blocks: more than 128 of them in each
    g, k = circulant(3000, 150, np.arange(150) % 7 + 1), 24
    og = to_oracle(g)
    hier, dist = ([2, 4, 3], [1, 10, 100]) if kind == "map" else (None, None)
    part = np.random.default_rng(8).integers(0, k, g.n).astype(np.uint32)
    obj = O.comm_cost(og, part, hier, dist) if hier else O.edge_cut(og, part)
    maxw, lmax = int(np.bincount(part).max()), 140
    want = O.jet_refine(og, k, lmax, False, 0, part, obj, maxw, hier, dist)
    with H.Context(0, 256 << 20) as c:
        for name, v in tunes.items():
            c.tune(name, v)
        got = c.jet_refine(c.upload(g), k, lmax, part, obj, maxw, hierarchy=hier, distance=dist)
    assert got[1:] == want[1:]
    np.testing.assert_array_equal(got[0], want[0])
