"""Fronts with many pivots: chains of reduced parts with 20 to 36 modes have fronts of 33
to 49 rows and 24 to 40 pivots, on either side of 32 pivots (one panel of a warp) and of 48
rows (the large fronts).  Solves with the Newton matrix have the backward error of a stable
factorisation, at most 10 n eps (|N| |x| + |b|) in the infinity norm (FP64), or agree with
the dense solution to 1e-8 as the other mixed-precision solves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("modes", [20, 24, 28, 30, 33, 36])
def test_solves(gpu, tmp_path, modes, mixed):
    from fedem_gb300 import models
    from fedem_gb300.batch import Batch, Model

    m = Model(*models.superelement_chain_c3(str(tmp_path), n_parts=4, n_modes=modes, steps=3)[:2])
    b = Batch([m], mixed=mixed)
    b.assemble_newton(0, 3.0e6, 2.0e3, 0.9)
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
