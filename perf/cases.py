"""Timed cases of the batched regional shortest-path engine.

A case is one request of a routing program to the engine, through the public
Python names over the C ABI: the graph of the device is resident, a set of
nets is planned into batches, and one pass prepares the batches from the
nets, relaxes them, reads the statuses and returns what the program asked for
(paths per target, label images, or edge gradients).  Graphs and net shapes
are those of the repository's configurations (`bfx.workloads`) and of the
same generator at odd sizes.

The resident graph of a generator specification is kept per process, as a
router keeps its device's graph over all its nets; nets, upstream gradients
and the plan come from the seed.
"""
import math
import os
import random
import sys
from collections import OrderedDict

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "bf-new_b200"))

import bfx  # noqa: E402
from bfx import expansion, workloads  # noqa: E402

# Generator specifications: the configurations' graphs, and "grid" (float
# costs) / "gridi" (integer costs) at the case's own tile grid and tile size.
# c3 is timed on 128x128 tiles (4.2M vertices, 42M edges).


def _spec(case):
    name = case["graph"]
    if name in ("grid", "gridi"):
        spec = dict(workloads.GRAPHS["c1f" if name == "grid" else "c1"])
        spec.update(tiles_x=case["tiles_x"], tiles_y=case["tiles_y"], nodes_per_tile=case["nodes"])
        return spec, (case["tiles_x"], case["tiles_y"])
    if name in ("c2", "c3small"):
        return workloads.bench_graph_spec(name)
    spec = dict(workloads.GRAPHS[name])
    return spec, (spec["tiles_x"], spec["tiles_y"])


_resident = OrderedDict()  # specification -> (layout, grid, resident graph, mean weight), at most 5


def _graph(case):
    spec, grid = _spec(case)
    key = repr(sorted(spec.items()))
    if key not in _resident:
        g, order, _ = bfx.synth_graph(**spec)
        layout = bfx.build_device_graph_layout(g, order)
        mean = float(np.mean(layout.arrays["csr_weights"], dtype=np.float64))
        _resident[key] = (layout, grid, bfx.ResidentDeviceGraph.upload_once(layout), mean)
        while len(_resident) > 5:
            _resident.popitem(last=False)  # states that still use it keep it alive
    _resident.move_to_end(key)
    return _resident[key]


def _nets(case, layout, grid, seed):
    """The case's nets: boxes of side U[lo, hi] tiles with U[1, targets]
    targets, then full-graph nets."""
    qs = []
    if case["nets"]:
        qs += workloads.box_queries(layout, grid, case["nets"], case["lo"], min(case["hi"], *grid), 7919 * seed + 11,
                                    targets=(1, case["targets"]))
    if case["full"]:
        qs += workloads.full_graph_queries(layout, grid, case["full"], 7919 * seed + 12, first_id=len(qs),
                                           targets_per_query=case["targets"])
    return qs


# kind: what the program asks for --
#   "paths"      prepare the planned batches, relax, statuses, paths per target
#   "gradients"  the same, then dL/dweight of every edge for L = sum of g_t * distance_t
#   "screen"     prepare on the device from the nets, relax, statuses, largest distance per batch and the
#                first net's label image
#   "labels"     one batch through an engine class, statuses and whole label images
#   "net"        one net through the per-query entry point, status and its label image
#   "expansion"  nets whose boxes miss targets, retried on larger regions
# engine: "frontier", "jacobi", "dense"; control: "persistent", "chunked", "per_round".
# step: near/far threshold step in mean edge weights (0: plain frontier, the
# default), pack: chunk slots per warp item -- the values the tuner picks for
# such sets, fixed here so that every pass asks for the same schedule.
_BASE = dict(nets=0, full=0, lo=0, hi=0, targets=1, width=32, engine="frontier", control="persistent", step=0.0,
             pack=4, tiles_x=0, tiles_y=0, nodes=0)


def _case(**kw):
    unknown = set(kw) - set(_BASE) - {"name", "kind", "graph"}
    if unknown:
        raise ValueError(f"unknown case fields {unknown}")
    return {**_BASE, **kw}


def listed():
    return [
        # an interactive query: one short net on a small device, latency and launches count
        _case(name="net_small", kind="net", graph="c1", nets=1, lo=8, hi=8, targets=4),
        # one long net over a whole large device: a single lane, no batch to hide its latency
        _case(name="net_device", kind="net", graph="c2", full=1),
        # a lookahead table: whole label images of eight sources (configuration c1)
        _case(name="labels_c1", kind="labels", graph="c1", full=8, width=8),
        # the synchronous pull engine on a batch of regional nets (Bellman-Ford semantics, uneven tiles)
        _case(name="labels_jacobi", kind="labels", graph="grid", tiles_x=29, tiles_y=31, nodes=45, nets=13, lo=6, hi=20,
              targets=2, width=16, engine="jacobi"),
        # the dense chaotic engine on a full-width batch
        _case(name="labels_dense", kind="labels", graph="gridi", tiles_x=23, tiles_y=37, nodes=70, nets=32, lo=8,
              hi=23, targets=2, width=32, engine="dense"),
        # a training step of a cost model (configuration c4): forward, paths, gradient of every edge weight
        _case(name="gradients_c4", kind="gradients", graph="c1f", nets=512, lo=8, hi=32, targets=32, step=4.0),
        # the headline batch (configuration c2): 256 uneven regional nets, tuned step
        _case(name="paths_c2", kind="paths", graph="c2", nets=256, lo=4, hi=64, step=4.0),
        # the same kind of nets with the options as they come: plain frontier
        _case(name="paths_c2_plain", kind="paths", graph="c2", nets=64, lo=4, hi=64, targets=8),
        # 32 full-graph sources in one batch (configuration c3 on 128x128 tiles)
        _case(name="paths_c3", kind="paths", graph="c3small", full=32, targets=32, step=1.0, pack=8),
        # very many small nets and a few long ones, screened for reachability before they are committed
        # (configuration c5 on 128x128 tiles)
        _case(name="screen_c5", kind="screen", graph="c3small", nets=1024, lo=2, hi=16, full=4, step=1.0, pack=8),
        # a host-polled run (a program that wants control between chunks of rounds), ragged tiles
        _case(name="paths_polled", kind="paths", graph="grid", tiles_x=61, tiles_y=47, nodes=53, nets=40, lo=5, hi=41,
              targets=3, width=16, control="chunked", step=4.0),
        # rip-up of short nets: many miss a target in their first box and are retried on larger ones
        _case(name="expansion", kind="expansion", graph="gridi", tiles_x=33, tiles_y=27, nodes=61, nets=96, lo=1, hi=3,
              targets=3),
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _grid(rng, most):
    """A generated grid of at most `most` vertices."""
    tx, ty = _log(rng, 9, 70), _log(rng, 9, 70)
    nodes = _log(rng, 17, 150)
    while tx * ty * nodes > most:
        if nodes > 17:
            nodes = max(17, nodes * 2 // 3)
        else:
            tx, ty = max(9, tx * 2 // 3), max(9, ty * 2 // 3)
    return dict(graph=rng.choice(("grid", "gridi")), tiles_x=tx, tiles_y=ty, nodes=nodes)


def draw(rng: random.Random):
    kind = rng.choice(("net", "labels", "gradients", "paths", "paths", "paths", "expansion"))
    if kind == "net":
        if rng.random() < 0.5:
            return _case(kind=kind, graph=rng.choice(("c2", "c3small")), full=1, targets=_log(rng, 1, 9))
        g = _grid(rng, 300_000)
        side = min(g["tiles_x"], g["tiles_y"])
        return _case(kind=kind, nets=1, lo=_log(rng, 2, side), hi=side, targets=_log(rng, 1, 9), **g)
    if kind == "labels":
        g = _grid(rng, 120_000)
        width = rng.choice((8, 16, 32))
        side = min(g["tiles_x"], g["tiles_y"])
        nets = rng.randint(1, width)
        lo = _log(rng, 2, side)
        return _case(kind=kind, nets=nets, lo=lo, hi=rng.randint(lo, side), targets=rng.randint(1, 4), width=width,
                     engine=rng.choice(("frontier", "jacobi", "dense")), **g)
    if kind == "gradients":
        g = _grid(rng, 120_000)
        side = min(g["tiles_x"], g["tiles_y"])
        lo = _log(rng, 2, side)
        return _case(kind=kind, nets=_log(rng, 16, 512), lo=lo, hi=rng.randint(lo, side), targets=_log(rng, 1, 32),
                     step=rng.choice((0.0, 2.0, 4.0)), width=rng.choice((8, 16, 32)), **g)
    if kind == "expansion":
        lo = rng.randint(1, 2)
        return _case(kind=kind, nets=_log(rng, 8, 96), lo=lo, hi=lo + rng.randint(0, 2), targets=rng.randint(1, 4),
                     width=rng.choice((8, 32)), **_grid(rng, 80_000))
    kind = rng.choice(("paths", "paths", "screen"))
    step, pack = rng.choice(((0.0, 4), (1.0, 8), (2.0, 4), (4.0, 4), (4.0, 2)))
    which = rng.randrange(4)
    if which == 0:
        lo = _log(rng, 2, 32)
        return _case(kind=kind, graph="c2", nets=_log(rng, 8, 256), lo=lo, hi=rng.randint(lo, 64), step=step, pack=pack,
                     targets=_log(rng, 1, 8), width=rng.choice((8, 32)))
    if which == 1:
        lo = _log(rng, 2, 12)
        return _case(kind=kind, graph="c3small", nets=_log(rng, 64, 1024), lo=lo, hi=rng.randint(lo, 16),
                     full=rng.randint(0, 4), step=step, pack=pack)
    if which == 2:
        return _case(kind=kind, graph=rng.choice(("c2", "c3small")), full=_log(rng, 2, 24), step=step or 2.0, pack=pack,
                     targets=_log(rng, 1, 32))
    g = _grid(rng, 300_000)
    side = min(g["tiles_x"], g["tiles_y"])
    lo = _log(rng, 2, side)
    return _case(kind=kind, nets=_log(rng, 2, 64), lo=lo, hi=rng.randint(lo, side), targets=rng.randint(1, 5),
                 control=rng.choice(("persistent", "chunked", "per_round")), step=step, pack=pack,
                 width=rng.choice((8, 16, 32)), **g)


_ENGINES = {"frontier": bfx.BatchedFrontierPushEngine, "jacobi": bfx.BatchedJacobiPullEngine,
            "dense": bfx.BatchedDenseChaoticPushEngine}
_CONTROLS = {"persistent": bfx.CONTROL_PERSISTENT, "chunked": bfx.CONTROL_CHUNKED, "per_round": bfx.CONTROL_PER_ROUND}


def prepare(case, seed):
    layout, grid, graph, mean = _graph(case)
    queries = _nets(case, layout, grid, seed)
    ws = bfx.Workspace(graph)
    s = {"kind": case["kind"], "stores": _stores(case), "layout": layout, "graph": graph, "ws": ws, "queries": queries,
         "options": bfx.GpuRunOptions(control_mode=_CONTROLS[case["control"]])}
    if case["kind"] == "labels":
        s["batch"] = bfx.make_description(layout, queries, case["width"])
        s["engine"] = _ENGINES[case["engine"]](graph, ws)
    elif case["kind"] == "expansion":
        s["expansion"] = expansion.ExpansionOptions(
            schedule_kind=expansion.DOUBLING, maximum_expansions=4,
            planner_policy=bfx.BatchPlannerPolicy(case["width"], 1, 8, 2, 1, narrow_lanes=True))
    else:
        # regional nets by overlap; full-graph nets alone share everything
        policy = (bfx.BatchPlannerPolicy(case["width"], 1, 8, 2, 1, narrow_lanes=True) if case["nets"]
                  else bfx.BatchPlannerPolicy(case["width"], 0, 1, 64, 1))
        plan = bfx.make_overlapping_batch_plan(layout, queries, policy)
        s["batches"] = plan.descriptions()
        if case["kind"] == "screen":
            s["lanes"] = bfx.QueryLanes.from_descriptions(plan.descriptions(), queries)
        if case["step"]:
            ws.set_batch_deltas([case["step"] * mean] * plan.batch_count)
        ws.set_chunk_pack(case["pack"])
        if case["kind"] == "gradients":
            total = sum(len(d.targets) for d in plan.descriptions())
            s["upstream"] = np.random.default_rng(seed).uniform(0.1, 1.0, total).astype(np.float32)
    return s


def _statuses(statuses):
    return np.array([[st.converged, st.reached_target_mask, st.bounding_box_miss_mask, st.stop_reason, st.error_bits]
                     for st in statuses], np.int64)


def _image(bits, predecessors):
    return {"distance": bits.view(np.float32), "predecessor": predecessors.view(np.int32)}


class _Store:
    """The program's result arrays, kept between requests: values of any
    length up to the capacity, the rest filled (-1, floats 0)."""

    def __init__(self, rows, dtype, columns=None):
        self.fill = 0 if np.dtype(dtype).kind == "f" else -1
        self.array = np.full(rows if columns is None else (rows, columns), self.fill, dtype)
        self.held = 0

    def put(self, values):
        n = len(values)
        self.array[:n] = values
        self.array[n:max(n, self.held)] = self.fill
        self.held = n
        return self.array


# Vertices of a path, per target: the longest on these graphs have about 60.
_PATH = 64
_PATH_FIELDS = {"target": np.int32, "selected_source": np.int32, "distance": np.float32, "path_length": np.int32,
                "reached": np.int32, "reconstruction": np.int32}


def _stores(case):
    nets = case["nets"] + case["full"]
    targets = nets * case["targets"]
    if case["kind"] == "expansion":
        return {"outcomes": _Store(nets, np.int64, len(expansion.OUTCOME_FIELDS)), "histogram": _Store(16, np.int64)}
    stores = {"status": _Store(nets, np.int64, 5), "bounds": _Store(nets, np.float32),
              "vertices": _Store(targets * _PATH, np.int32), "labels": _Store(targets * _PATH, np.float32),
              "edges": _Store(targets * _PATH, np.int32)}
    stores.update({f: _Store(targets, t) for f, t in _PATH_FIELDS.items()})
    return stores


def run(s):
    ws, put = s["ws"], s["stores"]
    if s["kind"] == "net":
        q = s["queries"][0]
        status = ws.run_query(q.sources, q.targets, q.selected_tiles, s["options"])
        return {"status": _statuses([status]), **_image(*ws.download_lane(0, 0))}
    if s["kind"] == "labels":
        statuses, labels = s["engine"].run_with_distances([s["batch"]], s["options"])
        return {"status": _statuses(statuses), **_image(*labels[0])}
    if s["kind"] == "expansion":
        got = expansion.run_expansion(ws, s["layout"], s["queries"], s["expansion"])
        regions = np.zeros((len(s["queries"]), s["layout"].tile_count), np.uint8)
        for i, tiles in enumerate(got["final_tiles"]):
            regions[i, tiles] = 1
        return {"outcomes": put["outcomes"].put([[o[f] for f in expansion.OUTCOME_FIELDS] for o in got["outcomes"]]),
                "histogram": put["histogram"].put(got["histogram"]), "regions": regions}
    if s["kind"] == "screen":
        ws.prepare_from_queries(s["lanes"])
        ws.execute(s["options"])
        return {"status": put["status"].put(_statuses(ws.fetch_statuses())),
                "bounds": put["bounds"].put(ws.label_bounds().view(np.float32)), **_image(*ws.download_lane(0, 0))}
    ws.prepare(s["batches"])
    ws.execute(s["options"])
    out = {"status": put["status"].put(_statuses(ws.fetch_statuses()))}
    paths = ws.compact_paths(raw=True)
    for f in _PATH_FIELDS:
        out[f] = put[f].put(paths["summaries"][f])
    for f, t in (("vertices", np.int32), ("labels", np.float32), ("edges", np.int32)):
        out[f] = put[f].put(paths[f].view(t))
    if s["kind"] == "gradients":
        out["gradient"] = ws.edge_usage_adjoint(s["upstream"])
    return out


def _edges(layout):
    a = layout.arrays
    src = np.repeat(np.arange(layout.vertex_count), np.diff(a["csr_row_offsets"].astype(np.int64)))
    return src, a["csr_destinations"].astype(np.int64), a["csr_weights"].astype(np.float64), a["owner_tiles"]


def _distances(layout, queries):
    """Distances of the nets' regional searches in 64 bits, one column per
    net: sweeps over all edges until nothing changes."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    src, dst, w, owner = _edges(layout)
    src, dst, w = (torch.from_numpy(x).to(dev) for x in (src, dst, w))
    inside = np.zeros((layout.tile_count, len(queries)), bool)
    d = torch.full((layout.vertex_count, len(queries)), math.inf, dtype=torch.float64, device=dev)
    for i, q in enumerate(queries):
        inside[q.selected_tiles, i] = True
        d[torch.from_numpy(q.sources.astype(np.int64)).to(dev), i] = 0.0
    inside = torch.from_numpy(inside[owner]).to(dev)
    admitted = inside[src] & inside[dst]
    at = dst[:, None].expand(-1, len(queries))
    while True:
        cand = torch.where(admitted, d[src] + w[:, None], math.inf)
        new = d.scatter_reduce(0, at, cand, "amin")
        if torch.equal(new, d):
            return d.cpu().numpy()
        d = new


def exact(case, seed):
    """Distances in 64 bits; the predecessor of a vertex and the vertices of a
    path depend on ties between 32-bit distances and have no such value."""
    layout, grid, _, _ = _graph(case)
    queries = _nets(case, layout, grid, seed)
    if case["kind"] == "expansion" or layout.edge_count * len(queries) > 300_000_000:
        return None
    if case["kind"] in ("labels", "net"):
        d = _distances(layout, queries)
        if case["kind"] == "net":
            return {"status": None, "distance": d[:, 0], "predecessor": None}
        image = np.full((layout.vertex_count, case["width"]), math.inf)
        image[:, :len(queries)] = d
        return {"status": None, "distance": image, "predecessor": None}
    by_net = {}
    for i in range(0, len(queries), 16):
        d = _distances(layout, queries[i:i + 16])
        for j, q in enumerate(queries[i:i + 16]):
            by_net[i + j] = d[:, j]
    order = [int(i) for b in prepare(case, seed)["batches"]
             for i in b.query_index_by_lane[:bin(b.valid_lane_mask).count("1")]]
    if case["kind"] == "screen":
        return {"status": None, "bounds": None, "distance": by_net[order[0]], "predecessor": None}
    out = dict.fromkeys(("status", "vertices", "labels", "edges", "gradient", *_PATH_FIELDS))
    out["distance"] = _Store((case["nets"] + case["full"]) * case["targets"], np.float64).put(
        np.concatenate([by_net[i][queries[i].targets.astype(np.int64)] for i in order]))
    return out


def work(case):
    """Every edge of the nets' regions read once (destination, weight, edge
    id), one 8-byte label per (vertex, net) of the regions written once, one
    addition and one comparison per (edge, net) -- regions at their mean size;
    label images and gradients written once."""
    spec, (tx, ty) = _spec(case)
    tiles, nodes, degree = tx * ty, spec["nodes_per_tile"], spec["intra"] + spec["inter"]
    side = (case["lo"] + min(case["hi"], tx, ty)) / 2
    box = min(side * side, tiles)
    if case["kind"] == "expansion":
        box = min((2 * side + 2) ** 2, tiles)  # boxes grow until the targets are inside
    covered = tiles if case["full"] else tiles * (1 - math.exp(-case["nets"] * box / tiles))
    lane_vertices = (case["nets"] * box + case["full"] * tiles) * nodes
    total = covered * nodes * degree * 12 + lane_vertices * 8
    if case["kind"] in ("net", "screen"):
        total += tiles * nodes * 8
    elif case["kind"] == "labels":
        total += tiles * nodes * case["width"] * 8
    elif case["kind"] == "gradients":
        total += tiles * nodes * degree * 4
    return {"bytes": int(total), "flops": int(2 * degree * lane_vertices)}


def tolerance(case):
    """Labels are minima of left-folded 32-bit sums and the predecessor is the
    smallest edge id among the edges that give the minimum: both are the same
    in every order of relaxation."""
    return "exact"
