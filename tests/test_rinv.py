"""The integer form of the softened pair factor (csrc/rinv.cuh).

On the CPU the host build of the header is compared with long double; on the
GPU the direct sum that uses it is compared with numpy long double.
Error budget of one factor, relative: final rounding 2^-53; delta rounded to
2^-54, times 3/2; the series rounded to 2^-53; U within 4 units of 2^-58, times
3/2: below 2^-51 together.
"""
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rinv") / "rinv_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", os.path.join(HERE, "rinv_check.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("scale,eps,inside", [(1.0, 0.0, True), (1.0, 0.005, True), (1e-3, 1e-4, True), (1e20, 1e17, True),
                                              (1e-40, 0.0, True), (1e-40, 1.0, True), (1e80, 0.5, True), (1e80, 0.0, True),
                                              (1e-75, 0.0, True), (1e95, 0.0, False), (1e-95, 0.0, False), (1e-95, 1e-95, False)])
def test_factor_against_long_double(exe, scale, eps, inside):
    r = subprocess.run([exe, repr(scale), repr(eps), "40000"], capture_output=True, text=True, check=True)
    f = r.stdout.split()
    v = dict(zip(f[0::2], f[1::2]))
    assert float(v["max3"]) <= 2.0 ** -51 and float(v["max1"]) <= 2.0 ** -51
    assert (int(v["out"]) == 0) == inside  # outside: the FP64 form takes over


@pytest.mark.gpu
@pytest.mark.parametrize("n,scale,eps", [(2, 1.0, 0.0), (33, 1.0, 0.01), (257, 1e20, 1e17), (300, 1e-30, 0.0), (300, 1e-95, 0.0),
                                         (1000, 1e3, 1e-3)])
def test_direct_sum_against_long_double(n, scale, eps):
    import vipp_gb300

    rng = np.random.default_rng(n)
    x = scale * rng.standard_normal((n, 3))
    with vipp_gb300.Solver(p=4, s=32, eps=eps, m=1.0 / n) as s:
        s.preprocess(x, np.zeros_like(x))
        a = s.direct_accel()
    d = x[None].astype(np.longdouble) - x[:, None].astype(np.longdouble)
    u = (d * d).sum(2) + np.longdouble(eps * eps)
    np.fill_diagonal(u, 1)
    t = d * (u ** np.longdouble(-1.5))[:, :, None] / n
    if float(np.abs(t).max()) > 1e300:  # beyond FP64: the sums overflow as the FP64 form's do
        assert not np.isfinite(a).all()
        return
    # one factor within 2^-51; a separation, a product and a sum rounded per term (the worst case of n sums), G m once
    tol = (2.0 ** -51 + (n + 4) * 2.0 ** -53) * np.abs(t).sum(1)
    assert (np.abs(a - t.sum(1)) <= tol.astype(np.float64)).all()
