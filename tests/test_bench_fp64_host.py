"""The bench line's FP64 roofline is given for the meshes whose kernels issue
the counted instructions: from the cell count on at which agx_plain.cu forms
products with integer instructions."""
import os
import re
import sys

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, REPO)

import bench  # noqa: E402


def test_fp64_roofline_only_where_its_counts_hold():
    with open(os.path.join(REPO, "anuga_core_gb300", "csrc", "agx_plain.cu")) as f:
        first = int(re.search(r"IMUL_MIN_CELLS = (\d+);", f.read()).group(1))
    assert bench.fp64_roofline(first - 1, 1.0, 525.0) is None
    roof = bench.fp64_roofline(first, 1.0, 525.0)
    assert abs(roof["achieved"] - bench.FP64_PER_CELL_STEP["lane_ops"] * first * 1.0e3 / 1.0e9) < 1.0e-9
    assert roof["peak"] == 525.0
