"""The figures of the committed captures that bench.py reads, and its launch count, without a GPU."""
import re
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))

import bench  # noqa: E402


@pytest.mark.parametrize("workload,capture", [("spheroid", "k_pass_gabriel_spheroid_1m.md"),
                                              ("sheet", "k_pass_polarity_sheet_100k.md")])
def test_roofline_figures_are_the_present_captures(workload, capture):
    # the instruction count and the DRAM bytes of the capture's text, per cell
    text = (ROOT / "profiles" / capture).read_text()
    cells = 1_000_000 if workload == "spheroid" else 100_000
    inst = bench.pass_profile(workload, "warp_inst_per_cell")
    counts = [float(m) * 1e6 / cells for m in re.findall(r"smsp__inst_executed.sum \| ([0-9.]+) M", text)]
    assert any(c == pytest.approx(inst, rel=1e-3) for c in counts), (inst, counts)
    dram = bench.traffic_per_pass(workload)
    read = [float(m) * 1e6 / cells for m in re.findall(r"([0-9.]+) MB", text)]
    assert any(r == pytest.approx(dram, rel=2e-3) for r in read), (dram, read)


def test_workloads_without_a_capture_have_no_traffic():
    assert bench.traffic_per_pass("small") is None
    assert bench.pass_profile("small", "warp_inst_per_cell") is None


def test_launches_of_a_call():
    source = (ROOT / "tecs_gb300" / "csrc" / "tecs_gpu.cu").read_text()
    assert int(re.search(r"constexpr int kSmallSteps = (\d+);", source).group(1)) == bench.SMALL_STEPS
    small = {"k_step_small": [1.0]}
    assert [bench.launches_per_call(small, 1, k) for k in (1, 32, 33, 100)] == [1, 1, 2, 4]
    assert bench.launches_per_call({"k_pass_heun1": [1.0], "k_scatter": [1.0]}, 8, 10) == 80
    assert "per step" in bench.roofline_kernel(small) and "per step" not in bench.roofline_kernel({"k_pass_euler": []})
