"""What relaxed a set's lanes, as the library reports it, and what follows from
it: the tuner does not choose between launches that are the same."""
import pytest

import bfx
from bfx import workloads
from test_gpu_resident import POLICY, graph

pytestmark = pytest.mark.gpu
FULL = bfx.BatchPlannerPolicy(32, 0, 1, 10000, 1, narrow_lanes=True)


def test_lanes_by_kernel(gpu):
    layout, grid = graph("c1f", 151, 157, 45)
    regional = bfx.make_overlapping_batch_plan(layout, workloads.box_queries(layout, grid, 20, 2, 30, seed=5),
                                               POLICY).descriptions()
    whole = bfx.make_overlapping_batch_plan(layout, workloads.full_graph_queries(layout, grid, 3, 6, first_id=20),
                                            FULL).descriptions()
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    ws = bfx.Workspace(resident)

    def used(descs, **options):
        ws.prepare(descs)
        if options.pop("engines", False):
            ws.set_batch_engines([b % 3 for b in range(len(descs))])
        ws.execute(bfx.GpuRunOptions(**options))
        assert all(s.stop_reason == bfx.STOP_CONVERGED for s in ws.fetch_statuses())
        k = ws.last_execute_kernels()
        assert all((n > 0) == (r > 0) for n, r in k.values()), k
        return tuple(n for n, _ in k.values())

    assert used(regional) == (20, 0, 0)
    assert used(whole) == (0, 3, 0)
    assert used(regional + whole) == (20, 3, 0)
    assert used(regional + whole, control_mode=bfx.CONTROL_CHUNKED) == (20, 3, 0)
    assert used(regional + whole, control_mode=bfx.CONTROL_PER_ROUND) == (0, 3, 20)
    assert used(regional, control_mode=bfx.CONTROL_CHUNKED, rounds_per_chunk=3) == (0, 0, 20)
    assert used(regional + whole, maximum_rounds=60_000) == (0, 0, 23)
    on_grid = sum(bin(d.valid_lane_mask).count("1") for b, d in enumerate(regional) if b % 3 != 2)
    assert used(regional, engine=bfx.ENGINE_AUTO, engines=True) == (20 - on_grid, 0, on_grid)
    ws.set_batch_engines([])
    ws.set_resident_nets(0)
    assert used(regional + whole) == (0, 0, 23)
    ws.close()
    resident.close()


def test_tuner_leaves_the_pack_of_searches(gpu):
    """Clusters and teams have no chunk slots, so there is nothing to time: the
    workspace keeps the pack it had.  Lanes on the grid still have it tuned."""
    layout, grid = graph("c1f", 32, 32, 64)
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    for seed in range(4):
        descs = bfx.make_overlapping_batch_plan(layout, workloads.box_queries(layout, grid, 12, 2, 20, seed=seed),
                                                POLICY).descriptions()
        ws = bfx.Workspace(resident)
        ws.set_chunk_pack(1)
        bfx.load().bfx_autotune_reset()
        ws.autotune(descs)
        ws.execute(bfx.GpuRunOptions(engine=bfx.ENGINE_AUTO))
        if ws.last_execute_kernels()["grid"][0] == 0:
            assert ws.chunk_pack() == 1
        ws.close()
    resident.close()
    bfx.load().bfx_autotune_reset()
