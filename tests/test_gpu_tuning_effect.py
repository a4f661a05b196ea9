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


@pytest.mark.parametrize("n,s,slices", [(1 << 17, 64, (1024, 2048, 4096)), (1 << 20, 512, (2048, 8192, 32768))])
def test_slice_lengths_differ(n, s, slices):
    """Slices no longer than n / 32, and lists of more sources than the shortest: every length sums the
    near field in an order of its own, within the mixed tolerance (RMS 2e-6, max 1e-4) of each other."""
    import vipp_gb300
    from vipp_gb300.workloads import plummer
    x, v = plummer(n, 2)
    got = []
    with vipp_gb300.Solver(p=4, s=s, eps=0.005, m=1.0 / n, precision="mixed") as sol:
        for length in slices:
            sol.set_tuning(p2p_slice=length)
            sol.preprocess(x, v)
            got.append(sol.accel())
    for k, a in enumerate(got):
        for b in got[:k]:
            e = np.linalg.norm(a - b, axis=1) / np.linalg.norm(b, axis=1)
            assert not np.array_equal(a, b) and np.sqrt(np.mean(e * e)) <= 2e-6 and e.max() <= 1e-4


@pytest.mark.parametrize("precision,p", [("mixed", 4), ("mixed", 8), ("fp64", 4)])
def test_blocks_beside_the_far_field_repeat(precision, p):
    """The far field beside 0 to 16 blocks per SM of the near field: bit-identical to the one-stream
    order, evaluation after evaluation."""
    import vipp_gb300
    from vipp_gb300.workloads import plummer
    n = 60_000
    x, v = plummer(n, 2)
    kw = dict(p=p, s=128, eps=0.01, m=1.0 / n, precision=precision)
    with vipp_gb300.Solver(flags=vipp_gb300.FLAG_SERIAL, **kw) as s:
        s.preprocess(x, v)
        ref = s.accel()
    with vipp_gb300.Solver(**kw) as s:
        s.preprocess(x, v)
        for conc in (0, 1, 2, 3, 4, 6, 8, 16):
            s.set_tuning(p2p_blocks_conc=conc)
            for _ in range(3):
                assert np.array_equal(s.accel(), ref)
