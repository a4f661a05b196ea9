"""The far field beside the near field on a shared SM: repeated evaluations are
bit-identical to the one-stream order (a tile of the M2M kernel used to be
cleared while its operator was being loaded, which warps slowed by the near
field's made visible)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,occ", [(100_000, 4, 6), (200_000, 4, 6), (100_000, 8, 8)])
def test_concurrent_evaluations_repeat(n, p, occ):
    import vipp_gb300
    from vipp_gb300.workloads import plummer
    x, v = plummer(n, 2)
    kw = dict(p=p, s=256, eps=0.01, m=1.0 / n, precision="mixed")
    with vipp_gb300.Solver(flags=vipp_gb300.FLAG_SERIAL, **kw) as s:
        s.preprocess(x, v)
        ref = s.accel()
    with vipp_gb300.Solver(**kw) as s:
        s.set_tuning(p2p_occupancy=occ)
        s.preprocess(x, v)
        for _ in range(10):
            assert np.array_equal(s.accel(), ref)
