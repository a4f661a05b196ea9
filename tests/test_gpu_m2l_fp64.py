"""The FP64 M2L (csrc/m2l_fp64.cu): every expansion order against the oracle,
tiles with few targets, and the form whose class groups run as blocks of their
own (small trees) bit-identical to the one-block form (a forest of more than
304 tiles)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", range(1, 11))
def test_split_and_whole_tiles_agree_and_match_the_oracle(p):
    import oracle
    import vipp_gb300

    rng = np.random.default_rng(p)
    sizes = np.concatenate([[450], rng.integers(300, 700, 44)])  # 45 systems: at least 360 tiles of one octant
    xs = [rng.standard_normal((n, 3)) * rng.uniform(0.5, 2.0, 3) for n in sizes]
    s, eps = 4, 0.01
    with vipp_gb300.Batch(sizes, p=p, s=s, eps=eps, masses=1.0 / sizes, precision="fp64") as b:
        b.upload(np.concatenate(xs), np.zeros((int(sizes.sum()), 3)))
        whole = b.accel()
    at = np.concatenate([[0], np.cumsum(sizes)])
    for k in (0, 1, 44):
        with vipp_gb300.Solver(p=p, s=s, eps=eps, m=1.0 / sizes[k], precision="fp64") as sol:
            sol.preprocess(xs[k], np.zeros_like(xs[k]))
            a = sol.accel()
        assert np.array_equal(a, whole[at[k]:at[k + 1]])
        ref = oracle.oracle().accel(xs[k], s, 1.0, 1.0 / sizes[k], eps, p)
        # the FP64 pipeline's tolerance against the oracle
        assert np.max(np.linalg.norm(a - ref, axis=1) / np.linalg.norm(ref, axis=1)) <= 1e-10
