"""bench.py's roofline of the Toeplitz CG: the operator's own bytes, and beside them
what its passes move with the vector updates that ride on them."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_updates_are_reported_beside_the_operator():
    sys.path.insert(0, ROOT)
    import bench
    P, nt, c = 384, 768, 8
    prof = {"toeplitz": (20.0, 33, 0.0), "spread": (2.0, 2, 0.0), "crop": (0.5, 1, 0.0)}
    _, roof, _ = bench.roofline_from_profile(prof, 6698.0, "measured", {"np": P, "nz": 256}, c, 1)
    # the passes in order: before the loop, the first step, nine more
    vectors = [0.5 + 1 + 2] + [2 + 2] + 9 * [5 + 2]
    moved = sum(c * (v * P * P + 4 * P * nt) for v in vectors) / 11
    w = roof["with_updates"]
    assert abs(w["bytes_per_unit"] - moved) <= 1
    assert abs(w["achieved"] - 11 * 256 * moved / 0.020 / 1e9) < 0.1
    assert abs(w["frac"] - w["achieved"] / 6698.0) < 1e-3
    # an NFFT group has none
    prof = {"spread": (27.0, 22, 0.0), "crop": (3.0, 11, 0.0)}
    _, roof, _ = bench.roofline_from_profile(prof, 6698.0, "measured", {"np": P, "nz": 256}, c, 1)
    assert "with_updates" not in roof
