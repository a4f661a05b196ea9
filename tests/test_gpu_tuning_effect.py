"""Tuning knobs take effect: what test_gpu_tuning.py compares really differs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def evaluated(n, tune, **kw):
    """Accelerations and kernel launches of one evaluation."""
    import vipp_gb300
    from vipp_gb300.workloads import plummer
    x, v = plummer(n, 2)
    with vipp_gb300.Solver(p=6, s=64, eps=0.005, m=1.0 / n, **kw) as s:
        s.set_tuning(**tune)
        s.preprocess(x, v)
        s.accel()  # buffers sized
        b = s.launch_count()
        a = s.accel()
        return a, s.launch_count() - b


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_blocks_beside_the_far_field_are_honoured(precision):
    """As many blocks beside the far field as in all (6 of 6) leave no second launch of the near
    field for afterwards; the library's own choice (8: 3 or 4) and 2 leave one. Same results."""
    few, with_rest = evaluated(30_000, {"p2p_blocks": 6, "p2p_blocks_conc": 2}, precision=precision)
    auto, auto_launches = evaluated(30_000, {"p2p_blocks": 6}, precision=precision)
    all_, without = evaluated(30_000, {"p2p_blocks": 6, "p2p_blocks_conc": 6}, precision=precision)
    assert without == with_rest - 1 and auto_launches == with_rest
    assert np.array_equal(few, auto) and np.array_equal(few, all_)
