"""The large-front kernels share a wave of fronts out over the whole GPU: how many
blocks a front gets, and how its panels of 32 pivots and tiles are cut, follows from
the sizes.  Frames whose fronts have 49 to 183 rows and 6 to 108 pivots (one panel,
exact panels of 32, a remainder, one block to many blocks a front, waves of one front
and of many) are stepped alone and all together, and must agree to the last bit; and a
linear solve with each one's Newton matrix must have the backward error of a stable
factorisation, at most 10 n eps (|N| |x| + |b|) in the infinity norm (FP64), or agree
with the dense solution to 1e-8 as the other mixed-precision solves (two refinement
sweeps)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(3, 1), (6, 1), (2, 2), (4, 2), (9, 2), (3, 3), (4, 4)]  # storeys, bays


def _frames():
    from fedem_gb300 import models
    from fedem_gb300.batch import Model

    return [Model(*models.space_frame_c2(seed=11, storeys=s, bays=b, n_joints=2, n_springs=2, steps=3))
            for s, b in SIZES]


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_alone_and_together_agree_bitwise(gpu, mixed):
    from fedem_gb300.batch import Batch

    ms = _frames()
    assert min(m.max_front for m in ms) > 48
    together = Batch(ms, mixed=mixed)
    assert together.run()["models_failed"] == 0
    for k, m in enumerate(ms):
        alone = Batch([m], mixed=mixed)
        assert alone.run()["models_failed"] == 0
        np.testing.assert_array_equal(together.triads(k), alone.triads(0))
        np.testing.assert_array_equal(together.norms(k), alone.norms(0))
        alone.close()
    together.close()


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_solves_have_a_small_backward_error(gpu, mixed):
    from fedem_gb300.batch import Batch

    for m in _frames():
        b = Batch([m], mixed=mixed)
        b.assemble_newton(0, 3.0e6, 0.0, 0.9)
        rp, ci = m.csr_pattern()
        n = np.zeros((m.neq, m.neq))
        vals = b.newton_values(0)
        for i in range(m.neq):
            n[i, ci[rp[i]:rp[i + 1]]] = vals[rp[i]:rp[i + 1]]
        assert b.factor(0) == 0
        rhs = np.random.default_rng(3).standard_normal((2, m.neq))
        x = b.solve(0, rhs)
        if mixed:
            xd = np.linalg.solve(n, rhs.T).T
            assert np.abs(x - xd).max() <= 1e-8 * np.abs(xd).max()
        else:
            scale = np.abs(n).sum(1).max() * np.abs(x).max() + np.abs(rhs).max()
            assert np.abs(x @ n - rhs).max() <= 10 * m.neq * 2.0**-53 * scale
        b.close()
