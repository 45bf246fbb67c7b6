"""The bench line's pair-kernel traffic: a capture of the kernel, box and skin
of the run, else nothing."""

import json
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))

import bench  # noqa: E402


def test_only_a_capture_of_this_kernel_and_workload_counts(tmp_path):
    f = tmp_path / "t.json"
    assert bench.pair_traffic(65536, 2.5, f) is None
    f.write_text("not json")
    assert bench.pair_traffic(65536, 2.5, f) is None
    captures = [{"molecules": 65536, "skin_A": 2.5, "dram_bytes_per_launch": 7}]
    f.write_text(json.dumps({"kernel": "k_pair4<0,0,1>", "captures": captures}))
    assert bench.pair_traffic(65536, 2.5, f) is None
    f.write_text(json.dumps({"kernel": "k_pair4<0,0,1>", "dram_bytes_per_launch_full_size": 44800000}))
    assert bench.pair_traffic(65536, 2.5, f) is None
    f.write_text(json.dumps({"kernel": bench.PAIR_KERNEL, "captures": captures}))
    assert bench.pair_traffic(65536, 2.5, f) == 7
    assert bench.pair_traffic(65536, 2.0, f) is None
    assert bench.pair_traffic(8192, 2.5, f) is None


def test_the_kept_record_is_of_the_present_kernel():
    record = json.loads((ROOT / "profiles" / "pair_kernel_traffic.json").read_text())
    assert record["kernel"] == bench.PAIR_KERNEL
    for run in record["captures"]:
        assert bench.pair_traffic(run["molecules"], run["skin_A"]) == run["dram_bytes_per_launch"] > 0
