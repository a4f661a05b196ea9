"""Kernel timers: a class counts once per evaluation, whatever number of parts its
stage is queued in (bench.py's rates per launch divide by it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,flags", [("fp64", 0), ("mixed", 0), ("mixed", "FLAG_M2L_BF16"), ("mixed", "FLAG_M2L_CUDA_CORES")])
@pytest.mark.parametrize("mode", ["ref", "accurate"])
def test_one_count_per_evaluation(precision, flags, mode):
    import vipp_gb300
    from vipp_gb300.workloads import plummer
    n = 5000
    x, v = plummer(n, 1)
    with vipp_gb300.Solver(p=4, s=32, eps=0.01, m=1.0 / n, precision=precision, mode=mode,
                           flags=getattr(vipp_gb300, flags) if flags else 0) as s:
        s.preprocess(x, v)
        s.accel()
        s.enable_timing(True)
        s.kernel_times()
        s.accel()
        one = s.kernel_times()
        s.solve(1e-4)
        step = s.kernel_times()
    classes = ["tree", "operators", "p2m_m2m", "m2l", "l2l_l2p", "p2p"] + (["soften"] if mode == "accurate" else [])
    for c in classes:
        assert one[c][1] == 1 and step[c][1] == 4 and one[c][0] > 0, c


def test_one_count_per_batch_evaluation():
    import vipp_gb300
    from vipp_gb300.workloads import plummer
    sizes = np.array([700, 1500, 300])
    xs, vs = zip(*[plummer(int(n), 1) for n in sizes])
    with vipp_gb300.Batch(sizes, p=4, s=32, eps=0.01, masses=1.0 / sizes, precision="mixed") as b:
        b.upload(np.concatenate(xs), np.concatenate(vs))
        b.step(1e-4)
        b.enable_timing(True)
        b.kernel_times()
        b.step(1e-4)
        k = b.kernel_times()
    assert all(k[c][1] == 4 for c in ("tree", "operators", "p2m_m2m", "m2l", "l2l_l2p", "p2p"))
