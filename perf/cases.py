"""Performance cases: the partitioning and mapping calls of this framework over the range of sizes it is used with.

A case is one call of a user's program through gpu_heipa.py. Every input is made from the seed: 2D grids, R-MAT graphs
and 3D random geometric graphs as bench.py and the tests draw them. All results are whole numbers that do not depend on
the order of execution, so every output has to stay exactly the same.

Kinds of calls:
  partition  Context.partition (graph in host memory: upload and download are part of the call)
  resident   Context.partition_graph (graph already on the device)
  map        Context.process_map (host graph)          map_resident  Context.process_map_graph
  refine     Context.jet_refine of a given partition   batch         Context.partition_batch of many host graphs
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-heipa_b200"))
import gpu_heipa as H  # noqa: E402

HIERARCHIES = {"4:8:6": ([4, 8, 6], [1, 10, 100]), "2:4:8": ([2, 4, 8], [1, 5, 50]), "8:16": ([8, 16], [1, 20])}


def listed():
    return [
        # the smallest requests of a stream: a solve is a chain of short launches
        {"name": "part_rgg_3k", "do": "partition", "graph": "rgg", "n": 3001, "degree": 10.0, "w": 10, "k": 8,
         "config": "default"},
        # the small benchmark configuration: unit weights, about eight coarsening levels
        {"name": "part_grid_65k", "do": "partition", "graph": "grid", "x": 256, "y": 256, "w": 0, "k": 16,
         "config": "default"},
        # small skewed graph with many blocks: hub rows on levels that fit in L2
        {"name": "part_rmat_65k", "do": "partition", "graph": "rmat", "scale": 16, "degree": 8, "w": 10, "k": 128,
         "config": "default"},
        # ordinary mesh-like request, odd size
        {"name": "part_rgg_200k", "do": "partition", "graph": "rgg", "n": 199999, "degree": 10.0, "w": 10, "k": 32,
         "config": "default"},
        # the quality configuration: about ten times the refinement rounds
        {"name": "ultra_rmat_65k", "do": "partition", "graph": "rmat", "scale": 16, "degree": 16, "w": 10, "k": 64,
         "config": "ultra"},
        # large mesh into the most blocks a request asks for
        {"name": "part_grid_2m", "do": "resident", "graph": "grid", "x": 1733, "y": 1201, "w": 10, "k": 512,
         "config": "default"},
        # the headline configuration
        {"name": "part_rmat_4m", "do": "resident", "graph": "rmat", "scale": 22, "degree": 16, "w": 10, "k": 64,
         "config": "default"},
        # a mapping request of a stream: 17 dependent and concurrent sub-solves
        {"name": "map_hm_rgg_70k", "do": "map", "graph": "rgg", "n": 70001, "degree": 10.0, "w": 100, "hier": "8:16",
         "config": "HM"},
        # integrated mapping: the J objective in every refinement round of one hierarchy
        {"name": "map_im_rgg_2m", "do": "map_resident", "graph": "rgg", "n": 2097151, "degree": 14.0, "w": 100,
         "hier": "4:8:6", "config": "IM"},
        # the mapping benchmark configuration, the largest input
        {"name": "map_hm_rgg_8m", "do": "map_resident", "graph": "rgg", "n": 8388608, "degree": 14.0, "w": 100,
         "hier": "4:8:6", "config": "HM"},
        # an existing partition brought up to date after changes: refinement of the input level alone
        {"name": "refine_grid_1m", "do": "refine", "graph": "grid", "x": 1024, "y": 1023, "w": 10, "k": 64,
         "moved": 0.05},
        # many small requests handed over at once
        {"name": "batch_32", "do": "batch", "count": 32, "n_lo": 1000, "n_hi": 200000, "w": 10, "workers": 16},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, n, w):
    kind = rng.choice(("grid", "rmat", "rgg"))
    if kind == "grid":
        x = max(2, int(round(math.sqrt(n * rng.uniform(1.0, 4.0)))))
        return {"graph": "grid", "x": x, "y": max(2, n // x), "w": w}
    if kind == "rmat":
        return {"graph": "rmat", "scale": max(4, int(round(math.log2(n)))), "degree": rng.choice((8, 16)), "w": w}
    return {"graph": "rgg", "n": n, "degree": rng.choice((10.0, 14.0)), "w": w}


def draw(rng):
    do = rng.choice(("partition", "partition", "partition", "ultra", "resident", "resident", "map", "map_resident",
                     "refine", "batch"))
    if do == "partition":
        c = _draw_graph(rng, _log_uniform(rng, 1000, 200000), rng.choice((0, 10)))
        return dict(c, do="partition", k=rng.choice((2, 4, 8, 16, 32, 64, 128, 256, 6, 48, 100)), config="default")
    if do == "ultra":
        c = _draw_graph(rng, _log_uniform(rng, 1000, 100000), rng.choice((0, 10)))
        return dict(c, do="partition", k=2 ** rng.randint(1, 8), config="ultra")
    if do == "resident":
        c = _draw_graph(rng, _log_uniform(rng, 200000, 3000000), rng.choice((0, 10)))
        return dict(c, do="resident", k=2 ** rng.randint(1, 9), config="default")
    if do == "map":
        c = _draw_graph(rng, _log_uniform(rng, 2000, 200000), 100)
        return dict(c, do="map", hier=rng.choice(sorted(HIERARCHIES)), config=rng.choice(("HM", "IM", "HM-ultra")))
    if do == "map_resident":
        c = _draw_graph(rng, _log_uniform(rng, 200000, 3000000), 100)
        return dict(c, do="map_resident", hier=rng.choice(sorted(HIERARCHIES)), config=rng.choice(("HM", "IM")))
    if do == "refine":
        c = _draw_graph(rng, _log_uniform(rng, 20000, 2000000), rng.choice((0, 10)))
        return dict(c, do="refine", k=2 ** rng.randint(1, 8), moved=round(rng.uniform(0.01, 0.1), 3))
    return {"do": "batch", "count": rng.randint(8, 40), "n_lo": 1000, "n_hi": 100000, "w": 10, "workers": 16}


# ---- inputs ---------------------------------------------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) % (1 << 62))
    return g


def _to_graph(n, keys, w, gen, explicit_vw):
    """The CSR of the undirected edges keys = u * n + v (u < v, distinct, sorted), weights uniform in [1, w] (w = 0:
    unit weights)."""
    u, v = keys // n, keys % n
    both = torch.cat((u * n + v, v * n + u))
    ew = None
    if w:
        ew = torch.randint(1, w + 1, (keys.numel(),), generator=gen, device="cuda", dtype=torch.int32).repeat(2)
    both, order = torch.sort(both)
    xadj = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    xadj[1:] = torch.cumsum(torch.bincount(both // n, minlength=n), 0)
    adj = (both % n).to(torch.int32).cpu().numpy().view(np.uint32)
    return H.Graph(xadj.to(torch.int32).cpu().numpy().view(np.uint32), adj,
                   None if ew is None else ew[order].cpu().numpy(), np.ones(n, np.int32) if explicit_vw else None)


def _grid(x, y, w, gen):
    ids = torch.arange(x * y, device="cuda").view(y, x)
    n = x * y
    keys = torch.cat(((ids[:, :-1] * n + ids[:, 1:]).flatten(), (ids[:-1] * n + ids[1:]).flatten()))
    return _to_graph(n, torch.sort(keys)[0], w, gen, False)


def _rmat(scale, degree, w, gen):
    n, e = 1 << scale, degree << scale
    u = torch.zeros(e, dtype=torch.int64, device="cuda")
    v = torch.zeros(e, dtype=torch.int64, device="cuda")
    for _ in range(scale):  # quadrant probabilities 0.57, 0.19, 0.19, 0.05
        r = torch.rand(e, generator=gen, device="cuda")
        u = 2 * u + (r >= 0.76)
        v = 2 * v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    perm = torch.randperm(n, generator=gen, device="cuda")
    u, v = perm[u], perm[v]
    keys = (torch.minimum(u, v) * n + torch.maximum(u, v))[u != v]
    return _to_graph(n, torch.unique(keys), w, gen, False)


def _rgg(n, degree, w, gen):
    """Points uniform in the unit cube, connected within the radius of the given mean degree."""
    r = (degree / ((n - 1) * 4.0 / 3.0 * math.pi)) ** (1.0 / 3.0)
    cells = max(1, int(1.0 / r))
    p = torch.rand(n, 3, generator=gen, device="cuda")
    c = (p * cells).long().clamp_(max=cells - 1)
    cell = (c[:, 2] * cells + c[:, 1]) * cells + c[:, 0]
    order = torch.argsort(cell)
    count = torch.bincount(cell, minlength=cells ** 3)
    start = torch.cumsum(count, 0) - count
    found = []
    for off in range(14):  # half of the 27 cells around one (the others see the pair from their side)
        d = (off % 3 - 1, off // 3 % 3 - 1, off // 9 - 1)
        x, y, z = c[:, 0] + d[0], c[:, 1] + d[1], c[:, 2] + d[2]
        inside = (x >= 0) & (x < cells) & (y >= 0) & (y < cells) & (z >= 0) & (z < cells)
        i = inside.nonzero().flatten()
        other = ((z * cells + y) * cells + x)[i]
        reps = count[other]
        first = torch.cumsum(reps, 0) - reps
        i = torch.repeat_interleave(i, reps)
        j = order[torch.arange(i.numel(), device="cuda") + torch.repeat_interleave(start[other] - first, reps)]
        near = ((p[i] - p[j]) ** 2).sum(1) < r * r
        if off == 13:  # a point's own cell: every pair once
            near &= i < j
        i, j = i[near], j[near]
        found.append(torch.minimum(i, j) * n + torch.maximum(i, j))
    return _to_graph(n, torch.unique(torch.cat(found)), w, gen, True)


def _graph(case, gen):
    if case["graph"] == "grid":
        return _grid(case["x"], case["y"], case["w"], gen)
    if case["graph"] == "rmat":
        return _rmat(case["scale"], case["degree"], case["w"], gen)
    return _rgg(case["n"], case["degree"], case["w"], gen)


def _batch_sizes(case, rng):
    sizes = np.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"]), case["count"])).astype(int)
    ks = 2 ** rng.integers(1, 9, case["count"])
    return [int(n) for n in sizes], [int(k) for k in ks]


def prepare(case, seed):
    gen = _gen(seed)
    st = {"case": case, "seed": int(seed) % 1000003}
    if case["do"] == "batch":
        # the sizes belong to the case, the graphs to the seed
        sizes, st["ks"] = _batch_sizes(case, np.random.default_rng(case["count"]))
        st["graphs"] = []
        for i, n in enumerate(sizes):
            if i % 3 == 0:
                g = _grid(max(2, int(math.sqrt(2 * n))), max(2, int(math.sqrt(n / 2))), case["w"], gen)
            elif i % 3 == 1:
                g = _rmat(max(4, round(math.log2(n))), 8, case["w"], gen)
            else:
                g = _rgg(n, 10.0, case["w"], gen)
            st["graphs"].append(g)
        st["ctx"] = H.Context(0, 24 << 30)
        return st
    g = _graph(case, gen)
    scale = 2 if case["do"] in ("map", "map_resident") else 1  # sub-solves run side by side in the free space
    ctx = st["ctx"] = H.Context(0, scale * H.arena_estimate(g.n, g.m, g.ew is not None, g.vw is not None))
    if case["do"] in ("partition", "map"):
        st["g"] = g
    else:
        st["dg"] = ctx.upload(g)
    if case["do"] == "refine":
        # contiguous id ranges, as a partition kept from an earlier state of the data, some vertices displaced
        part = (np.arange(g.n, dtype=np.int64) * case["k"] // g.n).astype(np.uint32)
        rng = np.random.default_rng(seed)
        at = rng.choice(g.n, int(case["moved"] * g.n), replace=False)
        part[at] = rng.integers(0, case["k"], len(at)).astype(np.uint32)
        st["part"] = part
        st["obj"] = ctx.edge_cut(st["dg"], part)
        st["maxw"] = int(np.bincount(part, minlength=case["k"]).max())
        st["lmax"] = int(math.ceil(1.03 * (g.n / case["k"])))
    return st


def run(st):
    case, ctx, seed = st["case"], st["ctx"], st["seed"]
    do = case["do"]
    if do == "partition":
        return ctx.partition(st["g"], case["k"], 0.03, case["config"], seed)
    if do == "resident":
        return ctx.partition_graph(st["dg"], case["k"], 0.03, case["config"], seed)
    if do in ("map", "map_resident"):
        hier, dist = HIERARCHIES[case["hier"]]
        if do == "map":
            return ctx.process_map(st["g"], hier, dist, 0.03, case["config"], seed)
        return ctx.process_map_graph(st["dg"], hier, dist, 0.03, case["config"], seed)
    if do == "refine":
        return ctx.jet_refine(st["dg"], case["k"], st["lmax"], st["part"], st["obj"], st["maxw"])
    out = ctx.partition_batch(st["graphs"], st["ks"], 0.03, "default", seed, workers=case["workers"])
    return [np.concatenate([part for part, _ in out]), np.array([cut for _, cut in out], np.int64)]


def _size(case):
    """(vertices, directed entries) of a case's graph, before duplicates are dropped."""
    if case["graph"] == "grid":
        n = case["x"] * case["y"]
        return n, 4 * n
    if case["graph"] == "rmat":
        return 1 << case["scale"], 2 * case["degree"] << case["scale"]
    return case["n"], int(case["n"] * case["degree"])


def work(case):
    """Bytes of the graph read once and of the labels written once; one addition for each entry and vertex."""
    if case["do"] == "batch":
        sizes, _ = _batch_sizes(case, np.random.default_rng(case["count"]))
        n, m, weighted = sum(sizes), sum(int(n * (4, 16, 10)[i % 3]) for i, n in enumerate(sizes)), True
    else:
        n, m = _size(case)
        weighted = case["w"] > 0
    has_vw = case.get("graph") == "rgg"
    return {"bytes": 4 * (n + 1) + 4 * m * (2 if weighted else 1) + (4 * n if has_vw else 0) + 4 * n, "flops": n + m}


def tolerance(case):
    return "exact"
