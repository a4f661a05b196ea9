"""Near-field ranges by a warp per leaf and by 4 lanes (csrc/tree.cu): trees on
both sides of the line (16 leaves per SM) in contexts of their own and in one
that held a much larger system before: same accelerations, FP64 within the 1e-10
of test_gpu_parity.py of the oracle's."""
import numpy as np
import pytest

import oracle as O
from treecmp import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,below", [(700, True), (90_000, True), (130_000, False)])
def test_both_sides_of_the_line_and_after_a_large_system(n, below):
    import torch
    import vipp_gb300
    from vipp_gb300.workloads import plummer
    x, v = plummer(n, 3)
    kw = dict(p=3, s=64, eps=0.01, m=1.0 / n, precision="fp64")
    with vipp_gb300.Solver(**kw) as s:
        s.preprocess(x, v)
        a = s.accel()
        line = 16 * torch.cuda.get_device_properties(0).multi_processor_count
        assert (s.stats()["nleaves"] <= line) == below
    with vipp_gb300.Solver(**kw) as s:
        s.init_plummer(1_000_000, 1, 10.0)
        s.accel()
        s.preprocess(x, v)
        b = s.accel()
    assert np.array_equal(a, b)
    ref = O.oracle().accel(x, 64, 1.0, 1.0 / n, 0.01, 3)
    assert np.max(rel_err(a, ref)) <= 1e-10
