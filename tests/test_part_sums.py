"""The scratch of the M2Ls' part sums (csrc/part_sums.h). After a failed allocation
nothing is held, so that a caller who goes back to a smaller order gets buffers
again instead of null pointers; and it is sized for the trees that can use it. No
GPU needed."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("parts") / "part_sums_check")
    subprocess.run(["g++", "-std=c++17", "-O1", os.path.join(HERE, "part_sums_check.cpp"), "-o", out], check=True)
    return out


def run(exe, *args):
    return subprocess.run([exe, *map(str, args)], capture_output=True, text=True, check=True).stdout.split()


def test_failed_growth_holds_nothing(exe):
    assert run(exe) == ["1", "1", "1"]


@pytest.mark.parametrize("n,leaf,nsys,rows,bound,limit,held", [
    (1, 181, 1, 32, 8, 304, 8), (131_071, 181, 1, 32, 376, 304, 304), (30_000, 181, 1, 32, 104, 304, 104),
    # leaves of 181: 9,768 of them (8 no targets) are 305 tiles of 32, one fewer 304 and a rest
    (9768 * 181, 181, 1, 32, 5000, 304, 0), (9767 * 181, 181, 1, 32, 5000, 304, 304),
    (16_777_216, 181, 1, 128, 11_500, 304, 0), (4_194_304, 181, 1, 128, 2880, 304, 304),
    # a forest's systems may be all above level 2
    (512 * 1400, 181, 512, 32, 9000, 304, 304), (512 * 40_000, 181, 512, 32, 60_000, 304, 0)])
def test_sized_for_the_trees_that_can_use_it(exe, n, leaf, nsys, rows, bound, limit, held):
    assert run(exe, n, leaf, nsys, rows, bound, limit) == [str(held)]
