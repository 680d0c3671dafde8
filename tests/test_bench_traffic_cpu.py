"""Which captured DRAM traffic the bench reports beside a launch: only what the kernel that runs it was seen to move."""
import json
import os

import bench

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_traffic_of_another_kernel_or_size_is_not_reported():
    table = {"dense fp8 1x2x3": {"kernel": "a", "dram_bytes_per_launch": 1.0},
             "grouped down (32 local experts": {"kernel": "a", "dram_bytes_per_launch": 2.0, "routed_rows": 1000}}
    assert bench.traffic_entry(table, "dense fp8 1x2x3", "a")["dram_bytes_per_launch"] == 1.0
    assert bench.traffic_entry(table, "dense fp8 1x2x3", "b") is None and bench.traffic_entry(table, "dense fp8 1x2x4", "a") is None
    launch = "grouped down (32 local experts, %d routed rows, N=1 K=2)"
    assert bench.traffic_entry(table, launch % 1040, "a")["dram_bytes_per_launch"] == 2.0
    assert bench.traffic_entry(table, launch % 1060, "a") is None and bench.traffic_entry(table, launch % 1000, "b") is None


def test_every_entry_names_the_kernel_of_its_capture():
    with open(os.path.join(ROOT, "profiles", "traffic.json")) as f:
        table = json.load(f)
    for entry in table.values():
        capture = entry["source"].split(":")[0].split(" ")[0]
        assert os.path.basename(capture).startswith(entry["kernel"] + "_") and os.path.exists(os.path.join(ROOT, capture)), entry
