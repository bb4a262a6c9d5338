"""The bench line's roofline for each kernel that can hold the largest share of a sweep (no GPU)."""
from __future__ import annotations

import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402
from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402

INSTS = [W.plain_instance(256, 100, 5.0, 2.84, 50.0) for _ in range(3)] + [W.plain_instance(64, 50, 5.0, 2.84, 50.0)]
PT_STEPS = 3 * 256 * 256 * 99


@pytest.mark.parametrize("kernel", ["group<256>", "resident<256>"])
def test_march_in_one_kernel_has_issue_and_fp32_rates(kernel):
    ms = 2.0
    r = bench.sweep_roofline({kernel: (1, ms, 32.0 * PT_STEPS), "setup": (1, 0.5, 1e6)}, INSTS, 152, 2000.0)
    assert r["kernel"] == kernel and r["share_of_step"] == pytest.approx(0.8)
    assert r["achieved"] == pytest.approx(32.0 * PT_STEPS / (ms * 1e-3) / 1e9)
    rate = PT_STEPS / (ms * 1e-3)
    # FP32: 20 log2(256^2) + 456 flops per grid point and z step
    assert r["fp32"]["frac"] == pytest.approx(776.0 * rate / (152 * 256 * 2e9))
    with open(os.path.join(ROOT, "profiles", "ncu_traffic.json")) as f:
        rec = json.load(f)[kernel]
    assert r["issue"]["frac"] == pytest.approx(rec["thread_inst_per_pt_step"] * rate / (152 * 128 * 2e9))
    assert r["bound"] == ("issue" if r["issue"]["frac"] > r["frac"] else "hbm")
    assert r["traffic"] == pytest.approx(3 * rec["bytes_per_solve"])


def test_streaming_passes_are_held_to_the_copy_rate():
    r = bench.sweep_roofline({"rows<256>": (10, 1.0, 10 * 32.0 * 3 * 65536), "cols<256>": (9, 0.8, 1e9)}, INSTS, 152, 2000.0)
    assert r["bound"] == "hbm" and r["issue"] is None and r["fp32"] is None
    with open(os.path.join(ROOT, "profiles", "ncu_traffic.json")) as f:
        assert r["traffic"] == pytest.approx(json.load(f)["rows<256>"]["bytes_per_point"] * 3 * 65536)


def test_unknown_kernel_has_no_counters():
    r = bench.sweep_roofline({"setup": (1, 1.0, 1e6)}, INSTS, 152, 2000.0)
    assert r["bound"] == "hbm" and r["traffic"] is None and r["issue"] is None and r["fp32"] is None
