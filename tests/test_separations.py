"""FP64 separations of thin systems (csrc/rinv.cuh): every component of an
acceleration as accurate as its own terms allow, whichever way the system is turned.

Budgets: between positions on the frame's grid a separation is exact and rounded
once, 2^-53 of each component; the direct sum takes components to a target off it
from 2^54 quanta on, half a quantum more, 5/4 2^-53. Factor: 2^-51 on the grid; off
it two position errors of half a quantum each on pairs of 2^53 quanta and more,
3 * 1.37 * 2^-53 on top, below 2^-50."""
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rinv") / "rinv_grid_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fsanitize=signed-integer-overflow,shift",
                    "-fsanitize-undefined-trap-on-error", os.path.join(HERE, "rinv_grid_check.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("offset", [0.0, 0.3])
@pytest.mark.parametrize("h", [1.0, 1e-2, 1e-3, 1e-6, 1e-9, 1e-12])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_components_against_long_double(exe, axis, h, offset):
    r = subprocess.run([exe, str(axis), repr(h), repr(offset)], capture_output=True, text=True, check=True)
    f = r.stdout.split()
    v = dict(zip(f[0::2], map(float, f[1::2])))
    assert v["near"] <= 1.0 and v["direct"] <= 1.25 and v["factor"] <= 1.0
    if offset or h == 1.0:  # off the coordinate planes nearly every pair is taken
        assert v["near_taken"] > 20 * v["near_left"] and v["direct_taken"] > 20 * v["direct_left"]


@pytest.mark.parametrize("offset", [0.5 / 0.91, 8 / 0.91, -8 / 0.91])
def test_differences_wrap(exe, offset):
    """Positions on both sides of a multiple of 2^63 quanta (an extent of 1/16 about 1/2, 8, -8): the build traps on
    signed overflow, and the separations are as exact as elsewhere."""
    r = subprocess.run([exe, "0", "0.06", repr(offset), "0.06"], capture_output=True, text=True, check=True)
    f = r.stdout.split()
    v = dict(zip(f[0::2], map(float, f[1::2])))
    assert v["wraps"] > 50_000 and v["near"] <= 1.0 and v["direct"] <= 1.25 and v["factor"] <= 1.0


@pytest.mark.gpu
@pytest.mark.parametrize("h,offset", [(1e-3, 0.0), (1e-6, 0.0), (1e-12, 0.0), (1e-6, 0.3)])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_sheets_against_long_double(axis, h, offset):
    import vipp_gb300

    n, eps = 700, 0.01
    x = np.random.default_rng(axis).uniform(-1, 1, (n, 3))
    x[:, axis] = offset + h * x[:, axis]
    d = x[None].astype(np.longdouble) - x[:, None].astype(np.longdouble)
    u = (d * d).sum(2) + np.longdouble(eps * eps)
    t = d * (u ** np.longdouble(-1.5))[:, :, None] / n
    # factor and separation as above, a product and a sum rounded per term, G m once
    tol = ((2.0 ** -50 + 1.25 * 2.0 ** -53 + (n + 4) * 2.0 ** -53) * np.abs(t).sum(1)).astype(np.float64)
    with vipp_gb300.Solver(p=4, s=n, eps=eps, m=1.0 / n) as s:  # one leaf: the near field is the sum
        s.preprocess(x, np.zeros_like(x))
        for a in (s.direct_accel(), s.accel()):
            assert (np.abs(a - t.sum(1)) <= tol).all()
