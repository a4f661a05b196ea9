"""The direct sum at separations whose inverse cube is outside FP64's range (1e103
and beyond, 1e-103 and below) while the accelerations are inside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,G", [(1e-105, 6.674e-11), (1e-120, 1.0), (1e104, 1.0), (1e110, 1e30)])
def test_accelerations_inside_the_range(scale, G):
    import vipp_gb300

    n = 8
    x = scale * np.array([[(k >> a) & 1 for a in range(3)] for k in range(n)], float) + 0.1 * scale * np.random.default_rng(3).random((n, 3))
    with vipp_gb300.Solver(p=4, s=32, eps=0.0, G=G, m=1.0 / n) as s:
        s.preprocess(x, np.zeros_like(x))
        a = s.direct_accel()
    d = x[None].astype(np.longdouble) - x[:, None].astype(np.longdouble)
    u = (d * d).sum(2)
    np.fill_diagonal(u, 1)
    t = d * (u ** np.longdouble(-1.5))[:, :, None] * np.longdouble(G) / n
    # the factor in FP64 (sum of squares, rsqrt and three products: 2^-49), a product and a sum rounded per term, G m once
    tol = ((2.0 ** -49 + (n + 4) * 2.0 ** -53) * np.abs(t).sum(1)).astype(np.float64)
    assert (np.abs(a - t.sum(1)) <= tol).all()
