"""Downloads into page-locked and partly page-locked memory, and from several
workspaces of one graph at once, on a thread each."""
import threading

import numpy as np
import pytest
import torch

import bfx
from bfx import workloads

pytestmark = pytest.mark.gpu


def label_image(ws, batch, bits, pred):
    bfx._check(bfx.load().bfx_download_labels(ws._h, bfx.u32(batch), bfx._ptr(bits), bfx._ptr(pred)))


@pytest.mark.parametrize("locked", ["all", "first half", "second half"])
def test_page_locked_outputs(gpu, locked):
    layout, grid = workloads.build_graph("c1")
    desc = bfx.make_description(layout, workloads.full_graph_queries(layout, grid, 8, 3), 8)
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    ws = bfx.Workspace(resident)
    ws.prepare([desc])
    ws.execute(bfx.GpuRunOptions())
    bits, pred = ws.download_labels(0, 8)
    n = bits.size
    if locked == "all":
        host = torch.full((2, n), -2, dtype=torch.int32, pin_memory=True)
        got = host.numpy().view(np.uint32)
        label_image(ws, 0, got[0], got[1])
    else:
        page = 4096
        raw = np.full(2 * n + 2 * page, 0xFFFFFFFE, np.uint32)
        start = (-raw.ctypes.data // 4) % (page // 4)
        got = raw[start:start + 2 * n].reshape(2, n)
        assert got.ctypes.data % page == 0 and n * 4 % (2 * page) == 0
        at = got.ctypes.data + (0 if locked == "first half" else n * 2)
        cudart = torch.cuda.cudart()
        assert int(cudart.cudaHostRegister(at, n * 2, 0)) == 0  # half of the first output
        label_image(ws, 0, got[0], got[1])
        assert int(cudart.cudaHostUnregister(at)) == 0
    np.testing.assert_array_equal(got[0].reshape(bits.shape), bits)
    np.testing.assert_array_equal(got[1].reshape(pred.shape), pred)
    ws.close()
    resident.close()


def test_workspaces_on_threads(gpu):
    """Four workspaces of one graph, each on its own thread and stream: regional
    sets (clusters), whole-graph sets (a team each), label images of many
    pieces and paths, all at once, with the results of one after another."""
    spec = dict(workloads.GRAPHS["c1f"])
    spec.update(tiles_x=160, tiles_y=160, nodes_per_tile=45)
    g, order, _ = bfx.synth_graph(**spec)
    layout = bfx.build_device_graph_layout(g, order)
    grid = (160, 160)
    regional = bfx.BatchPlannerPolicy(32, 1, 8, 2, 1, narrow_lanes=True)
    sets = []
    for k in range(4):
        if k >= 2:
            queries = workloads.full_graph_queries(layout, grid, 3, 9 + k, targets_per_query=5)
            policy = bfx.BatchPlannerPolicy(32, 0, 1, 10000, 1, narrow_lanes=True)
        else:
            queries = workloads.box_queries(layout, grid, 24, 2, 40, seed=k, targets=(1, 4))
            policy = regional
        sets.append(bfx.make_overlapping_batch_plan(layout, queries, policy).descriptions())
    resident = bfx.ResidentDeviceGraph.upload_once(layout)

    def one_pass(ws, descs):
        ws.prepare(descs)
        ws.execute(bfx.GpuRunOptions())
        assert all(s.stop_reason == bfx.STOP_CONVERGED for s in ws.fetch_statuses())
        paths = ws.compact_paths(raw=True)
        return [*ws.download_lane(0, 0), *ws.download_labels(len(descs) - 1, descs[-1].lane_width),
                paths["vertices"], paths["labels"], paths["edges"], ws.label_bounds()]

    alone = []
    for descs in sets:
        ws = bfx.Workspace(resident)
        alone.append(one_pass(ws, descs))
        ws.close()
    failures, start = [], threading.Barrier(4)

    def worker(k):
        try:
            ws = bfx.Workspace(resident)
            start.wait(60)
            for _ in range(6):
                for x, y in zip(one_pass(ws, sets[k]), alone[k], strict=True):
                    np.testing.assert_array_equal(x, y)
            ws.close()
        except BaseException as e:  # noqa: BLE001 -- reported by the test
            failures.append((k, e))

    threads = [threading.Thread(target=worker, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not failures, failures
    resident.close()


def test_workspace_counts_its_buffers(gpu):
    """The buffers that a workspace keeps from one call to the next are in its
    reported bytes: the image buffer, the path buffer, the adjoint's."""
    layout, grid = workloads.build_graph("c1")
    desc = bfx.make_description(layout, workloads.full_graph_queries(layout, grid, 8, 3), 8)
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    ws = bfx.Workspace(resident)
    ws.prepare([desc])
    ws.execute(bfx.GpuRunOptions())
    held = [ws.device_bytes()]
    bits, _ = ws.download_labels(0, 8)
    held.append(ws.device_bytes())
    targets = len(ws.compact_paths())
    held.append(ws.device_bytes())
    ws.edge_usage_adjoint(np.ones(targets, np.float32))
    held.append(ws.device_bytes())
    grown = np.diff(held)
    assert grown[0] >= bits.nbytes and grown[1] >= targets * 28 and grown[2] >= layout.edge_count * 4
    ws.close()
    resident.close()


def test_large_payload_is_not_kept(gpu):
    """6.7 million path vertices (80 MB): the payload's buffer is the call's
    own, a small one stays with the workspace."""
    n, targets = 22_400, 300
    i = np.arange(n)
    e = n - 1
    g = bfx.InputGraph(i // 128, np.zeros(n), np.ones(n), np.zeros(n), i[:-1], i[1:], np.ones(e), np.zeros(e),
                       np.zeros(e), np.arange(e))
    layout = bfx.build_device_graph_layout(g, bfx.SpatialOrderConfig(0, 0, 1, 1))
    order = np.argsort(layout.tiles["new_to_old"])
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    ws = bfx.Workspace(resident)
    for count in (3, targets):
        q = bfx.RouteQuery(1, [int(order[0])], [int(v) for v in order[n - count:]], np.arange(layout.tile_count))
        ws.prepare([bfx.make_description(layout, [q], 1)])
        ws.execute(bfx.GpuRunOptions())
        before = ws.device_bytes()
        paths = ws.compact_paths(raw=True)
        lengths = paths["summaries"]["path_length"].astype(np.int64)
        assert sorted(lengths) == list(range(n - count, n))
        ends = np.cumsum(lengths + 1)
        np.testing.assert_array_equal(paths["labels"][ends - 1], lengths)
        np.testing.assert_array_equal(paths["vertices"][:lengths[0] + 1], order[:lengths[0] + 1])
        kept = ws.device_bytes() - before
        # the path buffer holds the targets' trails and the search's scratch
        if count == targets:
            assert len(paths["vertices"]) * 12 > 64 << 20 and kept < 16 << 20
    ws.close()
    resident.close()
