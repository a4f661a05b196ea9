"""Separations from fixed-point positions (csrc/rinv.cuh pair_fixed), against long double.

Budgets: the factor as in test_rinv.py, 2^-51; a position rounded to half a quantum
at each end and the rounding to 53 bits, for separations of 53 bits of quanta and
more: 2 * 2^-53 of the largest component. No factor of the FP64 form's tests is
refused: pairs too close for the frame take the FP64 difference (the GPU cases:
clumps, planes, coincident points, offsets, softening far above the extent)."""
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rinv") / "rinv_fixed_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", os.path.join(HERE, "rinv_fixed_check.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("scale,offset,eps,frames", [(1, 0, 0, True), (1, 0, 0.01, True), (1, 10, 0.01, True), (1, 0, 1, True), (1, 0, 3, True),
                                                     (1, 0, 1e3, False), (1e-3, 1, 1e-2, True), (1e20, 0, 1e17, True), (1e-40, 1e-38, 0, True),
                                                     (1, 1e9, 0, True), (1, 0, 1e-9, True), (1e95, 0, 0, False), (1e-95, 0, 0, False)])
def test_pairs_against_long_double(exe, scale, offset, eps, frames):
    r = subprocess.run([exe, repr(float(scale)), repr(float(offset)), repr(float(eps)), "100"], capture_output=True, text=True, check=True)
    f = r.stdout.split()
    v = dict(zip(f[0::2], f[1::2]))
    assert float(v["factor"]) <= 2.0 ** -51 and float(v["separation"]) <= 2.0 ** -52
    assert (int(v["frames"]) == 100) == frames and (int(v["taken"]) > 50 * int(v["left"])) == frames


def test_factor_beside_powers_of_two(tmp_path):
    out = str(tmp_path / "rinv_edge_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", os.path.join(HERE, "rinv_edge_check.cpp"), "-o", out], check=True)
    assert float(subprocess.run([out], capture_output=True, text=True, check=True).stdout) <= 2.0 ** -51


def cloud(kind, n, rng):
    x = rng.standard_normal((n, 3))
    if kind == "clump":  # separations down to 1e-12 of the extent
        x[::3] = x[0] + 1e-9 * rng.standard_normal((len(x[::3]), 3))
        x[1::7] = 1e-12 * rng.standard_normal((len(x[1::7]), 3))
    if kind == "plane":
        x[:, 2] = 0.25
    if kind == "coincident":
        x[::5] = x[0]
    if kind == "lattice":  # many separations beside powers of two
        x = np.round(4 * x) / 4 + 1e-5 * np.arange(n)[:, None]
    if kind == "offset":
        x = x * 1e-6 + 1e3
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["cloud", "clump", "plane", "coincident", "lattice", "offset"])
@pytest.mark.parametrize("n,eps", [(300, 0.0), (301, 1e-3), (700, 30.0)])
def test_sums_against_long_double(n, eps, kind):
    import vipp_gb300

    if kind == "coincident" and eps == 0.0:
        pytest.skip("unsoftened coincident points have no field")
    x = cloud(kind, n, np.random.default_rng(n))
    d = x[None].astype(np.longdouble) - x[:, None].astype(np.longdouble)
    u = (d * d).sum(2) + np.longdouble(eps * eps)
    np.fill_diagonal(u, 1)
    t = d * (u ** np.longdouble(-1.5))[:, :, None] / n
    # factor within 2^-51, separation within 2^-52, a product and a sum rounded per term, G m once; a
    # component's separation error is of the pair's largest component
    big = np.abs(t).max(2)
    tol = ((2.0 ** -51 + 2.0 ** -52 + (n + 4) * 2.0 ** -53) * big.sum(1))[:, None].astype(np.float64)
    with vipp_gb300.Solver(p=4, s=n, eps=eps, m=1.0 / n) as s:  # one leaf: the near field is the sum
        s.preprocess(x, np.zeros_like(x))
        for a in (s.direct_accel(), s.accel()):
            assert (np.abs(a - t.sum(1)) <= tol).all()
