"""CPU checks of what bench.py sets against the HBM roofline: algorithmic bytes
only for launches of the grid-wide kernels, a capture's DRAM bytes for sets
searched by clusters alone, nothing for what no figure covers."""
import pytest

from test_bench_helpers import REPO, load_bench


def kernels(clusters=0, teams=0, grid=0):
    return {"clusters": (clusters, 63), "teams": (teams, 63), "grid": (grid, 80)}


def test_grid_wide_launches_keep_their_algorithmic_bytes():
    bench = load_bench()
    moved, what, traffic, source, ceiling = bench.roofline_bytes("c2", kernels(grid=256), 123, 10 ** 8, 20.0, "4",
                                                                 "chunked")
    assert (moved, what) == (123, "algorithmic bytes")
    assert (traffic, source, ceiling) == bench.traffic_estimate("c2", 10 ** 8, 20.0, "4")
    moved, what, traffic, _, _ = bench.roofline_bytes("c2", kernels(grid=256), 123, 10 ** 8, 20.0, "4", "tiled")
    assert (moved, what, traffic) == (123, "algorithmic bytes", None)


def test_cluster_sets_use_their_captures():
    bench = load_bench()
    rows = [line.split() for line in (REPO / "profiles" / "search_traffic.txt").read_text().splitlines()
            if not line.startswith("#")]
    assert rows
    for _, dram, relaxations, step, summary in rows:
        assert (REPO / "profiles" / summary).exists()
        moved, what, traffic, source, ceiling = bench.roofline_bytes(
            "c2", kernels(clusters=256), 123, 2 * int(relaxations), 10.0, step, "chunked")
        assert moved == traffic == pytest.approx(2 * int(dram), rel=1e-9)
        assert "capture" in what and summary in source and ceiling is None
    moved, what, traffic, source, _ = bench.roofline_bytes("c2", kernels(clusters=256), 123, 10 ** 8, 10.0, "0.5",
                                                           "chunked")
    assert (moved, what, traffic) == (None, "not defined", None) and "not scaled" in source


@pytest.mark.parametrize("workload,used", [("c3", kernels(teams=64)), ("c5", kernels(clusters=4096, teams=16)),
                                           ("c2", kernels(clusters=200, grid=56)), ("c3small", kernels(clusters=3))])
def test_no_figure_where_none_was_captured(workload, used):
    moved, what, traffic, source, ceiling = load_bench().roofline_bytes(workload, used, 123, 10 ** 8, 10.0, "1",
                                                                        "chunked")
    assert (moved, what, traffic, ceiling) == (None, "not defined", None, None) and source
