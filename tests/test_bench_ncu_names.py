"""The committed ncu summary, which feeds the bench line's roofline.traffic,
holds kernels of the present code only, and one for every scope of the mixed
step whose kernel has another name."""
import glob
import json
import os
import re
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


def test_the_summary_is_of_the_present_kernels():
    src = "".join(open(f).read() for f in glob.glob(os.path.join(ROOT, "game_archived_gb300", "csrc", "gpu", "*.cu*")))
    present = set(re.findall(r"__global__[^;{]*?\b(k\w+)\s*\(", src))
    with open(bench.PROFILE_JSON) as f:
        captured = set(json.load(f)["kernels"])
    assert captured <= present, captured - present
    for scope, names in bench.NCU_NAMES.items():
        assert captured & set(names), scope
