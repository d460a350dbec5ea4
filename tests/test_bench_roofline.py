"""The BFS line's roofline entry counts what the kernel that ran reads: lists
for the default kernel, tiles for the b1-MMA slice test."""
import json

import numpy as np

import bench


def test_list_bytes():
    levels = np.full(20, 0xFFFFFFFF, dtype=np.uint32)
    assert bench.list_bytes(levels) == 0
    levels[[0, 3, 19]] = [0, 1, 2]
    assert bench.list_bytes(levels) == 36


def test_over_lists_the_bound_is_not_hbm():
    # RMAT-24: 8.9 M reached vertices, 0.383 ms, 256 MB of DRAM traffic
    r = bench.bfs_roofline(True, 12 * 8.9e6, 0.383e-3, 255.8e6, 6546.6, "measured")
    assert r["bound"] == "latency" and r["algorithmic_bytes_per_launch"] == 106_800_000
    assert r["achieved"] == round(106.8e6 / 0.383e-3 / 1e9, 1) and r["frac"] == round(106.8e6 / 0.383e-3 / 6546.6e9, 4)
    assert r["dram_gbs"] == round(255.8e6 / 0.383e-3 / 1e9, 1) and r["dram_frac"] < 0.2
    assert "dram_frac" not in bench.bfs_roofline(True, 1e6, 1e-3, None, 6546.6, "measured")


def test_over_tiles_as_before():
    r = bench.bfs_roofline(False, 2.4e9, 0.5e-3, 255.8e6, 6546.6, "measured")
    assert r["bound"] == "hbm" and r["achieved"] == 4800.0 and r["frac"] == round(4800 / 6546.6, 4)
    assert r["traffic"] is None and "dram_frac" not in r  # the capture is of the list kernel


def test_traffic_entries_say_how():
    for name, e in json.loads((bench.ROOT / "profiles" / "traffic.json").read_text()).items():
        assert name in bench.WORKLOADS and e["bytes_per_launch"] > 0 and len(e["how"]) > 40
        assert "algorithmic bytes per launch" not in e["how"]
