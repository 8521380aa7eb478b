"""Limits of a relaxation: a spent wall-clock budget ends every search the
normal way, with a status that says so and a workspace that stays usable, and a
round limit that a search could reach is kept exactly."""
import numpy as np
import pytest

import bfx

pytestmark = pytest.mark.gpu


def chain(n, tile=128):
    """Vertices 0 .. n-1 in tiles of `tile`, edges i -> i+1 of weight 1: the
    search from vertex 0 takes n rounds and reaches n-1 at distance n-1."""
    i = np.arange(n)
    e = n - 1
    g = bfx.InputGraph(i // tile, np.zeros(n), np.ones(n), np.zeros(n), i[:-1], i[1:], np.ones(e), np.zeros(e),
                       np.zeros(e), np.arange(e))
    layout = bfx.build_device_graph_layout(g, bfx.SpatialOrderConfig(0, 0, 1, 1))
    order = np.argsort(layout.tiles["new_to_old"])  # old vertex -> new
    q = bfx.RouteQuery(1, [int(order[0])], [int(order[n - 1])], np.arange(layout.tile_count))
    return layout, bfx.make_description(layout, [q], 1), order


def prepared(layout, desc):
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    ws = bfx.Workspace(resident)
    ws.prepare([desc])
    ws.set_batch_deltas([np.inf])
    return resident, ws


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [2_000, 3_000, 20_000, 450_000, 600_000, 900_000])
def test_spent_budget_stops_every_search(gpu, n, mode):
    """One block, clusters of 2 to 16 blocks, a team and the grid-wide kernel:
    a cluster's blocks stop in the same round, or they would wait for one
    another."""
    layout, desc, order = chain(n)
    resident, ws = prepared(layout, desc)
    ws.set_resident_nets(mode)
    ws.set_launch_budget(1)
    ws.execute(bfx.GpuRunOptions())
    (st,) = ws.fetch_statuses()
    assert st.stop_reason == bfx.STOP_FAILURE and st.converged == 0
    assert st.rounds_completed <= 256
    ws.set_launch_budget(30_000_000_000)
    if n <= 20_000:
        ws.execute(bfx.GpuRunOptions())
        (st,) = ws.fetch_statuses()
        assert st.stop_reason == bfx.STOP_CONVERGED
        assert ws.download_lane(0, 0)[0].view(np.float32)[order[n - 1]] == n - 1
    else:
        ws.execute(bfx.GpuRunOptions(maximum_rounds=2))
        assert ws.fetch_statuses()[0].stop_reason == bfx.STOP_MAXIMUM_ROUNDS
    for bad in (0, 30_000_000_001):
        with pytest.raises(ValueError):
            ws.set_launch_budget(bad)
    ws.close()
    resident.close()


def test_budget_covers_queued_searches(gpu):
    """More searches than run at once: each alone is well within the budget,
    all of them one after another are not."""
    layout, _, order = chain(20_000)
    first, last = int(order[0]), int(order[-1])
    queries = [bfx.RouteQuery(k, [first], [last], np.arange(layout.tile_count)) for k in range(32)]
    desc = bfx.make_description(layout, queries, 32)
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    ws = bfx.Workspace(resident)
    ws.prepare([desc] * 40)
    ws.execute(bfx.GpuRunOptions())
    assert all(st.stop_reason == bfx.STOP_CONVERGED for st in ws.fetch_statuses())
    together = ws.last_execute_timing()[0] * 1e6
    ws.set_launch_budget(int(0.6 * together))
    ws.execute(bfx.GpuRunOptions())
    assert all(st.stop_reason == bfx.STOP_FAILURE for st in ws.fetch_statuses())
    ws.prepare([desc])
    ws.execute(bfx.GpuRunOptions())
    assert ws.last_execute_timing()[0] * 1e6 < 0.6 * together
    assert ws.fetch_statuses()[0].stop_reason == bfx.STOP_CONVERGED
    ws.close()
    resident.close()


@pytest.mark.parametrize("limit,stop", [(65_536, "limit"), (69_999, "limit"), (70_000, "converged"),
                                        (70_100, "converged"), (1 << 40, "converged")])
def test_round_limit_that_a_search_can_reach(gpu, limit, stop):
    """A chain of 70,000 vertices takes 70,000 rounds (the last finds nothing
    to improve): limits below it stop the run there, whatever kernel would
    take the lane."""
    n = 70_000
    layout, desc, order = chain(n)
    resident, ws = prepared(layout, desc)
    ws.execute(bfx.GpuRunOptions(maximum_rounds=limit))
    (st,) = ws.fetch_statuses()
    bits, pred = ws.download_lane(0, 0)
    distance = bits.view(np.float32)[order]
    if stop == "converged":
        assert st.stop_reason == bfx.STOP_CONVERGED and st.rounds_completed <= limit
        np.testing.assert_array_equal(distance, np.arange(n))
    else:
        assert st.stop_reason == bfx.STOP_MAXIMUM_ROUNDS and st.rounds_completed == limit
        assert st.converged == 0 and st.active_lane_mask == 1
        np.testing.assert_array_equal(distance[:limit + 1], np.arange(limit + 1))
        assert np.all(np.isinf(distance[limit + 1:]))
        assert np.all(pred[order[1:limit + 1]] != 0xFFFFFFFF)
    ws.close()
    resident.close()
