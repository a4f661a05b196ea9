"""The scratch of the M2Ls' part sums (csrc/part_sums.h) after a failed allocation:
nothing is held, so that a caller who goes back to a smaller order gets buffers
again instead of null pointers. No GPU needed."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_failed_growth_holds_nothing(tmp_path):
    out = str(tmp_path / "part_sums_check")
    subprocess.run(["g++", "-std=c++17", "-O1", os.path.join(HERE, "part_sums_check.cpp"), "-o", out], check=True)
    assert subprocess.run([out], capture_output=True, text=True, check=True).stdout.split() == ["1", "1", "1"]
