"""Host-polled control of the cluster and team searches: launches of at most
rounds_per_chunk rounds (one, per round) with a look of the host after each,
whose state between the launches gives the labels of an uninterrupted search,
bit for bit."""
import ctypes as C

import numpy as np
import pytest

import bfx
from bfx import workloads
from test_gpu_limits import chain
from test_gpu_resident import POLICY, graph, relax

pytestmark = pytest.mark.gpu


def host_checks(ws):
    stats = (C.c_uint64 * 21)()  # bfx_device_work_statistics
    bfx._check(bfx.load().bfx_fetch_work_statistics(ws._h, stats, None))
    return stats[5]


def compare(layout, descs, step, controls, teams=False):
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    whole = relax(resident, descs, 1, step)
    for control, k in controls:
        ws = bfx.Workspace(resident)
        ws.prepare(descs)
        if step is not None:
            ws.set_batch_deltas([step] * len(descs))
        for _ in range(2):  # the second run starts from the first one's buffers
            ws.execute(bfx.GpuRunOptions(control_mode=control, rounds_per_chunk=k))
            statuses = ws.fetch_statuses()
            for b, d in enumerate(descs):
                got = ws.download_labels(b, d.lane_width)
                np.testing.assert_array_equal(got[0], whole[1][b][0])
                np.testing.assert_array_equal(got[1], whole[1][b][1])
        assert [{f: v for f, v in s.as_dict().items() if f != "rounds_completed"} for s in statuses] == whole[0]
        rounds = max(s.rounds_completed for s in statuses)
        per = 1 if control == bfx.CONTROL_PER_ROUND else k
        on_grid = ws.last_execute_kernels()["grid"][0]  # clusters from four rounds a launch on, teams always
        lanes = 0 if teams or per >= 4 else sum(bin(d.valid_lane_mask).count("1") for d in descs)
        assert on_grid == lanes
        checks = host_checks(ws)
        assert checks >= -(-rounds // per)
        if k >= 100_000 and control == bfx.CONTROL_CHUNKED:
            assert checks == 1
        ws.close()
    resident.close()


CHUNKED, PER_ROUND = bfx.CONTROL_CHUNKED, bfx.CONTROL_PER_ROUND


@pytest.mark.parametrize("step", [None, 3.0])
@pytest.mark.parametrize("nodes", [17, 32, 45, 70, 128, 300])
def test_tile_sizes(gpu, nodes, step):
    """The words of a net between launches: tiles below a word, of one, two,
    three, four and ten."""
    layout, grid = graph("c1f", 19, 23, nodes)
    queries = workloads.box_queries(layout, grid, 24, 1, 19, seed=nodes, targets=(1, 4))
    descs = bfx.make_overlapping_batch_plan(layout, queries, POLICY).descriptions()
    compare(layout, descs, step, [(PER_ROUND, 8), (CHUNKED, 3), (CHUNKED, 4), (CHUNKED, 5), (CHUNKED, 100_000)])


@pytest.mark.parametrize("side", [4, 20, 45, 64, 80, 110])
def test_net_sizes(gpu, side):
    """One block to the largest clusters."""
    layout, grid = graph("c1", 160, 160, 32)
    queries = workloads.box_queries(layout, grid, 1, side, side, seed=side, targets=(3, 3))
    descs = bfx.make_overlapping_batch_plan(layout, queries, POLICY).descriptions()
    compare(layout, descs, 40.0, [(PER_ROUND, 8), (CHUNKED, 4), (CHUNKED, 7)])


@pytest.mark.parametrize("step", [None, 3.0])
@pytest.mark.parametrize("lanes,nodes", [(1, 45), (12, 45), (20, 33)])
def test_whole_graph_lanes(gpu, lanes, nodes, step):
    """Teams: fewer lanes than teams and more, so that a launch ends in the
    middle of a lane and between two."""
    layout, grid = graph("c1f", 151, 157, nodes)
    queries = workloads.full_graph_queries(layout, grid, lanes, 9, targets_per_query=5)
    descs = bfx.make_overlapping_batch_plan(layout, queries, bfx.BatchPlannerPolicy(32, 0, 1, 10000, 1,
                                                                                   narrow_lanes=True)).descriptions()
    compare(layout, descs, step, [(PER_ROUND, 8), (CHUNKED, 11), (CHUNKED, 100_000)], teams=True)


def test_other_engines_beside_the_searches(gpu):
    """Per-batch engines: their batches are polled on the grid, the others in
    clusters."""
    layout, grid = graph("c2", 24, 24, 128)
    queries = workloads.box_queries(layout, grid, 24, 2, 20, seed=11)
    descs = bfx.make_overlapping_batch_plan(layout, queries, POLICY).descriptions()
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    reference = relax(resident, descs, 0)
    ws = bfx.Workspace(resident)
    ws.prepare(descs)
    ws.set_batch_engines([b % 3 for b in range(len(descs))])
    ws.execute(bfx.GpuRunOptions(engine=bfx.ENGINE_AUTO, control_mode=CHUNKED, rounds_per_chunk=4))
    assert all(s.stop_reason == bfx.STOP_CONVERGED for s in ws.fetch_statuses())
    for b, d in enumerate(descs):
        got = ws.download_labels(b, d.lane_width)
        np.testing.assert_array_equal(got[0], reference[1][b][0])
        np.testing.assert_array_equal(got[1], reference[1][b][1])
    ws.close()
    resident.close()


@pytest.mark.parametrize("n", [3_000, 900_000])
def test_spent_budget(gpu, n):
    """A cluster's and a team's polled run past the budget."""
    layout, desc, _ = chain(n)
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    ws = bfx.Workspace(resident)
    ws.prepare([desc])
    ws.set_launch_budget(1)
    ws.execute(bfx.GpuRunOptions(control_mode=CHUNKED, rounds_per_chunk=5))
    (st,) = ws.fetch_statuses()
    assert st.stop_reason == bfx.STOP_FAILURE and st.rounds_completed <= 5
    ws.close()
    resident.close()
