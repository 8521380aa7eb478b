"""Results on their way to the host: paths longer than the edges a summaries
pass keeps per target, weights over many orders of magnitude (the step of the
searches grows), and label images around the pieces that a download is cut
into."""
import numpy as np
import pytest

import bfx
from bfx import workloads
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def chain(n):
    """Vertices 0 .. n-1 in rows of ten per tile, edges i -> i+1 with weights
    2^-20 .. 2^20 and a costly shortcut over every third vertex."""
    i = np.arange(n)
    src = np.concatenate([i[:-1], i[:-3:3]])
    dst = np.concatenate([i[1:], i[3::3][:len(i[:-3:3])]])
    weight = np.concatenate([2.0 ** (i[:-1] % 41 - 20.0), np.full(len(i[:-3:3]), 2.0 ** 22)])
    e = len(src)
    g = bfx.InputGraph(i // 10, np.zeros(n), np.ones(n), np.zeros(n), src, dst, weight, np.zeros(e), np.zeros(e),
                       np.arange(e))
    return bfx.build_device_graph_layout(g, bfx.SpatialOrderConfig(0, 0, 1, 1))


@pytest.mark.parametrize("mode", [0, 1])
def test_long_paths_and_spread_weights(gpu, mode):
    """127, 128, 129 and 399 edges: within, at and beyond a trail."""
    layout = chain(400)
    order = np.argsort(layout.tiles["new_to_old"])  # old vertex -> new
    targets = [int(order[k]) for k in (5, 127, 128, 129, 399)]
    q = bfx.RouteQuery(1, [int(order[0])], targets, np.arange(layout.tile_count))
    desc = bfx.make_description(layout, [q], 1)
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    ws = bfx.Workspace(resident)
    ws.set_resident_nets(mode)
    ws.prepare([desc])
    ws.execute(bfx.GpuRunOptions())
    paths = ws.compact_paths()
    bits, pred = ws.download_labels(0, 1)
    grads = np.linspace(0.5, 2.0, len(paths)).astype(np.float32)
    gradient = ws.edge_usage_adjoint(grads)
    ws.close()
    resident.close()
    orc = Oracle.from_layout(layout)
    dist, opred = orc.region_sssp(q.sources, q.targets, q.selected_tiles)
    np.testing.assert_array_equal(bits[:, 0], dist)
    np.testing.assert_array_equal(pred[:, 0], opred)
    expect = np.zeros(layout.edge_count)
    for p, g in zip(paths, grads):
        st, verts, edges = orc.compact_path(q.sources, q.targets, q.selected_tiles, dist, p["target"])
        assert st == 0 and p["reconstruction"] == 0
        np.testing.assert_array_equal(p["vertices"], verts)
        np.testing.assert_array_equal(p["edges"], edges)
        np.testing.assert_array_equal(p["labels"].view(np.uint32), dist[verts])
        np.add.at(expect, edges, float(g))  # at most five float32 addends: exact in float64
    np.testing.assert_array_equal(gradient, expect.astype(np.float32))
    assert max(p["path_length"] for p in paths) == 399


@pytest.mark.parametrize("tiles,nodes,width", [((32, 32), 128, 1), ((32, 32), 127, 8), ((33, 31), 129, 8),
                                               ((8, 8), 20, 32)])
def test_label_images(gpu, tiles, nodes, width):
    """Images of exactly one piece of 512 KB, a little less and more, many
    pieces, and one small piece: the whole-batch image equals the lanes', and a
    lane equals the oracle's; a null output is left out."""
    spec = dict(workloads.GRAPHS["c1"])
    spec.update(tiles_x=tiles[0], tiles_y=tiles[1], nodes_per_tile=nodes)
    g, order, _ = bfx.synth_graph(**spec)
    layout = bfx.build_device_graph_layout(g, order)
    queries = workloads.full_graph_queries(layout, tiles, min(width, 5), 3)
    desc = bfx.make_description(layout, queries, width)
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    ws = bfx.Workspace(resident)
    ws.prepare([desc])
    ws.execute(bfx.GpuRunOptions())
    bits, pred = ws.download_labels(0, width)
    for lane in range(width):
        lane_bits, lane_pred = ws.download_lane(0, lane)
        np.testing.assert_array_equal(bits[:, lane], lane_bits)
        np.testing.assert_array_equal(pred[:, lane], lane_pred)
    only = np.empty(layout.vertex_count * width, np.uint32)
    bfx._check(bfx.load().bfx_download_labels(ws._h, bfx.u32(0), None, bfx._ptr(only)))
    np.testing.assert_array_equal(only.reshape(pred.shape), pred)
    assert ws.label_bounds()[0] == bits[bits < 0x7F800000].max()
    ws.close()
    resident.close()
    q = queries[0]
    dist, opred = Oracle.from_layout(layout).region_sssp(q.sources, q.targets, q.selected_tiles)
    np.testing.assert_array_equal(bits[:, 0], dist)
    np.testing.assert_array_equal(pred[:, 0], opred)
