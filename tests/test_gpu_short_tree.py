"""Trees at the edges of the one-block sort (at most 4,096 keys) and of the rule
that gives every leaf a warp (one grid of them, 9,728 cells on 152 SMs): tree,
member order and lists bit-exact with the oracle's, FP64 accelerations, which
read the near-field ranges, to the 1e-10 of test_gpu_parity.py."""
import numpy as np
import pytest

import oracle as O
from treecmp import canon_gpu, canon_ref, diff_trees, rel_err

pytestmark = pytest.mark.gpu


def points(n, kind):
    x, v = O.plummer_reference(n, 0.01, n)
    if kind == "lattice":  # keys that repeat: their order is the order of the particles
        x = np.round(x * 4) / 4 + 1e-5 * np.arange(n)[:, None]
    return x, v


@pytest.mark.parametrize("kind", ["plummer", "lattice"])
@pytest.mark.parametrize("n,s", [(1, 4), (2, 1), (33, 4), (257, 8), (1024, 16), (1025, 16), (4095, 32), (4096, 8), (4097, 8),
                                 (20_000, 16), (60_000, 8)])
def test_small_trees_and_ranges(n, s, kind):
    import vipp_gb300
    x, v = points(n, kind)
    orc = O.oracle()
    ref = canon_ref(orc.tree(x, s))
    a_ref = orc.accel(x, s, 1.0, 1.0 / n, 0.01, 2)
    with vipp_gb300.Solver(p=2, s=s, eps=0.01, m=1.0 / n) as sol:
        sol.preprocess(x, v)
        for _ in range(2):  # the second with the sorted key levels fitted to the tree
            a = sol.accel()
            assert diff_trees(canon_gpu(sol.tree_dump()), ref) == []
            scale = np.abs(a_ref).max()
            ok = np.linalg.norm(a_ref, axis=1) > 1e-6 * scale
            assert np.max(rel_err(a[ok], a_ref[ok]), initial=0.0) <= 1e-10
