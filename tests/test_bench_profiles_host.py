"""The FP64 instruction counts that bench.py's roofline reads from the committed ncu
summary: the reference's own additions, subtractions and products per cell, about 200 a
pass, with quotients, roots and powers of two in integers."""
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))
import bench  # noqa: E402


def test_fp64_pipe_counts():
    inst = bench.profile_table("fp64_pipe_inst_per_cell")
    for pass_ in ("flux", "stage"):
        assert 100 < inst[(pass_, "f64")] < 300
