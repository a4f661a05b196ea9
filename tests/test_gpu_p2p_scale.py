"""The mixed near field of a system as large as FP32 squares allow (1e18): tight
pairs of particles on a line, whose accelerations are their partner's. The sources
that fill up a batch must add nothing there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("newton", [False, True])
@pytest.mark.parametrize("at", [2e17, 1e18, 3e18])
def test_pairs_on_a_line(at, newton):
    import vipp_gb300

    sep = 3e12  # r^-3 = 3.7e-38, a normal FP32 number
    base = at * np.array([-1.0, -0.5, 0.25, 1.0])
    x = np.zeros((8, 3))
    x[:4, 0], x[4:, 0] = base, base + sep * np.array([1, -1, 1, -1])
    with vipp_gb300.Solver(p=4, s=16, eps=0.0, G=1.0, m=1.0, precision="mixed",
                           flags=vipp_gb300.FLAG_P2P_NEWTON if newton else 0) as s:
        s.preprocess(x, np.zeros_like(x))
        a = s.accel()
    d = x[None] - x[:, None]
    r = np.sqrt((d * d).sum(2))
    np.fill_diagonal(r, np.inf)
    ref = (d / r[:, :, None] ** 3).sum(1)
    # a coordinate is held to half an FP32 unit of `at` on either side of a pair: twice that in r^-2
    tol = 2 * 2.0 ** -24 * 2 * at / sep + 1e-3
    assert np.isfinite(a).all() and (np.abs(a - ref) <= tol * np.abs(ref).max()).all()
