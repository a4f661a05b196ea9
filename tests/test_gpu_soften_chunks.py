"""The softening correction's FP32 kernel at leaf sizes on both sides of its chunk
and lane-group edges (a leaf of one chunk, several, more than one pass of three),
against the oracle's accurate mode at test_gpu_accurate.py's mixed tolerance
(RMS 2e-6, max 1e-4). The softening is wide, so that the correction is ~1e-2 of
the field and a lost or doubled record shows."""
import math

import numpy as np
import pytest

import oracle as O
from treecmp import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s,n", [(4, 3000), (16, 3001), (21, 6000), (33, 6001), (70, 8000), (100, 12_001), (400, 30_000)])
@pytest.mark.parametrize("serial", [False, True])
def test_leaf_sizes_match_oracle(s, n, serial):
    import vipp_gb300
    x, v = O.plummer_reference(n, 0.05, s)
    ref = O.oracle().accel(x, s, 1.0, 1.0 / n, 0.05, 8, mode=1)
    with vipp_gb300.Solver(p=8, s=s, eps=0.05, m=1.0 / n, precision="mixed", mode="accurate",
                           flags=vipp_gb300.FLAG_SERIAL if serial else 0) as sol:
        sol.preprocess(x, np.zeros_like(x))
        e = rel_err(sol.accel(), ref)
    assert math.sqrt(np.mean(e * e)) <= 2e-6 and np.max(e) <= 1e-4
