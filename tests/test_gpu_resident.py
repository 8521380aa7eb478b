"""Searches outside the grid-wide kernels (bfx_set_resident_nets): the lanes
that fit a thread-block cluster's shared memory are relaxed there, larger
whole-graph lanes by a team of blocks each.  Their labels must be
the oracle's and the grid-wide kernels', bit for bit, for tiles of one word,
whole runs of words and ragged sizes, for nets from one block to clusters of
16, beside lanes that stay grid-wide in the same launch, and in every control
mode."""
import numpy as np
import pytest

import bfx
from bfx import workloads
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
POLICY = bfx.BatchPlannerPolicy(32, 1, 8, 2, 1, narrow_lanes=True)


def graph(base, tiles_x, tiles_y, nodes):
    spec = dict(workloads.GRAPHS[base])
    spec.update(tiles_x=tiles_x, tiles_y=tiles_y, nodes_per_tile=nodes)
    g, order, _ = bfx.synth_graph(**spec)
    return bfx.build_device_graph_layout(g, order), (tiles_x, tiles_y)


def relax(resident, descs, mode, step=None, **options):
    ws = bfx.Workspace(resident)
    ws.set_resident_nets(mode)
    ws.prepare(descs)
    if step is not None:
        ws.set_batch_deltas([step] * len(descs))
    ws.execute(bfx.GpuRunOptions(**options))
    statuses = [{k: v for k, v in s.as_dict().items() if k != "rounds_completed"} for s in ws.fetch_statuses()]
    labels = [ws.download_labels(b, d.lane_width) for b, d in enumerate(descs)]
    launches = ws.last_launch_count()
    ws.close()
    return statuses, labels, launches


def compare(layout, queries, descs, step=None, lanes=8, **options):
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    wide = relax(resident, descs, 0, step)
    here = relax(resident, descs, 1, step, **options)
    resident.close()
    assert here[0] == wide[0] and all(s["stop_reason"] == bfx.STOP_CONVERGED for s in here[0])
    for a, b in zip(here[1], wide[1]):
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[1], b[1])
    orc, done = Oracle.from_layout(layout), 0
    for b, d in enumerate(descs):
        for lane, qi in enumerate(d.query_index_by_lane[:bin(d.valid_lane_mask).count("1")]):
            if done < lanes:
                q = queries[int(qi)]
                dist, pred = orc.region_sssp(q.sources, q.targets, q.selected_tiles)
                np.testing.assert_array_equal(here[1][b][0][:, lane], dist)
                np.testing.assert_array_equal(here[1][b][1][:, lane], pred)
                done += 1
    return here[2], wide[2]


@pytest.mark.parametrize("step", [None, 3.0])
@pytest.mark.parametrize("nodes", [17, 32, 45, 70, 128, 300])
def test_tile_sizes(gpu, nodes, step):
    """Tiles below a word, of one word, of two (a power of two), of three
    (ragged runs), of one run of four, and of ten words."""
    layout, grid = graph("c1f", 19, 23, nodes)
    queries = workloads.box_queries(layout, grid, 40, 1, 19, seed=nodes, targets=(1, 4))
    descs = bfx.make_overlapping_batch_plan(layout, queries, POLICY).descriptions()
    compare(layout, queries, descs, step)


@pytest.mark.parametrize("side", [4, 20, 45, 64, 80, 110, 124, 160])
def test_net_sizes(gpu, side):
    """One net per launch: side^2 x 32 vertices take one block to the largest
    clusters; the two largest (with their tables of one-word tiles) do not fit
    and stay grid-wide."""
    layout, grid = graph("c1", 160, 160, 32)
    queries = workloads.box_queries(layout, grid, 1, side, side, seed=side, targets=(3, 3))
    descs = bfx.make_overlapping_batch_plan(layout, queries, POLICY).descriptions()
    here, wide = compare(layout, queries, descs, 40.0, lanes=1)
    # init, seed, one relaxation launch, finalize, either way
    assert here == wide == 4


@pytest.mark.parametrize("step", [None, 3.0, 200.0])
@pytest.mark.parametrize("lanes,nodes", [(1, 45), (7, 64), (12, 45), (20, 33)])
def test_whole_graph_lanes(gpu, lanes, nodes, step):
    """Whole-graph lanes that no cluster holds, one team of blocks each: lane
    widths 1, 8, 16 and 32, fewer lanes than teams and more, vertex counts that
    are and are not a multiple of a word, weights of zero."""
    layout, grid = graph("c1f", 151, 157, nodes)
    rng = np.random.default_rng(lanes)
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    a = layout.arrays
    weights = np.zeros(layout.edge_count, np.float32)
    weights[a["csr_edge_ids"]] = a["csr_weights"]
    weights[rng.integers(0, layout.edge_count, 2000)] = 0.0
    resident.set_weights(weights)
    a["csr_weights"] = weights[a["csr_edge_ids"]]
    a["csc_weights"] = weights[a["csc_edge_ids"]]
    queries = workloads.full_graph_queries(layout, grid, lanes, 9, targets_per_query=5)
    descs = bfx.make_overlapping_batch_plan(layout, queries, bfx.BatchPlannerPolicy(32, 0, 1, 10000, 1,
                                                                                   narrow_lanes=True)).descriptions()
    wide = relax(resident, descs, 0, step)
    for options in ({}, {"instrumentation": 1}):
        here = relax(resident, descs, 1, step, **options)
        assert here[0] == wide[0] and all(s["stop_reason"] == bfx.STOP_CONVERGED for s in here[0])
        for x, y in zip(here[1], wide[1]):
            np.testing.assert_array_equal(x[0], y[0])
            np.testing.assert_array_equal(x[1], y[1])
    resident.close()
    orc = Oracle.from_layout(layout)
    q = queries[int(descs[0].query_index_by_lane[0])]
    dist, pred = orc.region_sssp(q.sources, q.targets, q.selected_tiles)
    np.testing.assert_array_equal(here[1][0][0][:, 0], dist)
    np.testing.assert_array_equal(here[1][0][1][:, 0], pred)


@pytest.mark.parametrize("control", [bfx.CONTROL_PERSISTENT, bfx.CONTROL_CHUNKED, bfx.CONTROL_PER_ROUND])
def test_mixed_with_grid_wide_lanes(gpu, control):
    """Small nets beside full-graph lanes too large for a cluster, and both in
    one batch; counters of an instrumented run cover both paths."""
    layout, grid = graph("c1", 170, 170, 32)
    queries = workloads.box_queries(layout, grid, 30, 2, 30, seed=5) + \
        workloads.full_graph_queries(layout, grid, 3, 6, first_id=30)
    for policy in (POLICY, bfx.BatchPlannerPolicy(32, 0, 1, 10000, 1)):
        descs = bfx.make_overlapping_batch_plan(layout, queries, policy).descriptions()
        compare(layout, queries, descs, 60.0, lanes=4, control_mode=control)
        compare(layout, queries, descs, None, lanes=0, control_mode=control, instrumentation=1)


def test_other_engines_and_options_stay_grid_wide(gpu):
    """Per-batch engines beside resident nets; a round limit, an explicit grid
    and a kernel option keep every lane grid-wide (launch counts tell)."""
    layout, grid = graph("c2", 24, 24, 128)
    queries = workloads.box_queries(layout, grid, 24, 2, 20, seed=11)
    descs = bfx.make_overlapping_batch_plan(layout, queries, POLICY).descriptions()
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    reference = relax(resident, descs, 0)
    ws = bfx.Workspace(resident)
    ws.prepare(descs)
    ws.set_batch_engines([b % 3 for b in range(len(descs))])
    ws.execute(bfx.GpuRunOptions(engine=bfx.ENGINE_AUTO))
    assert all(s.stop_reason == bfx.STOP_CONVERGED for s in ws.fetch_statuses())
    for b, d in enumerate(descs):
        got = ws.download_labels(b, d.lane_width)
        np.testing.assert_array_equal(got[0], reference[1][b][0])
        np.testing.assert_array_equal(got[1], reference[1][b][1])
    ws.set_batch_engines([])
    for options in ({"maximum_rounds": 60000}, {"grid_policy": 1, "blocks_per_wgp": 1}, {"instrumentation": 2}):
        ws.execute(bfx.GpuRunOptions(**options))
        assert ws.last_launch_count() == 4
    ws.set_flat_items(3)
    ws.execute(bfx.GpuRunOptions())
    assert ws.last_launch_count() == 4
    with pytest.raises(ValueError):
        ws.set_resident_nets(2)
    ws.close()
    resident.close()
