"""Damped and quasi-static chains on the small batches' element and Newton kernels (four
lanes per beam) and on the large batches' (one thread): the same operations in the same
order, so alone and beside six long chains they agree to the last bit (tolerance zero).
Rayleigh damping gives the damping matrix and the filtered deformation rate; quasi-static
steps the passes without inertia, nonlinear and pure linear, and the change to dynamics."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(n, damped=False, **kw):
    from fedem_gb300 import models

    fsi = models.beam_chain_fsi(n, 0.25, 0.1, 0.01, clamp=0, load_node=n, load_dof=2,
                                load=0.0 if "motion" in kw else 90.0, **models.STEEL, **kw)
    if damped:
        assert "  elPropId = 1\n" in fsi
        fsi = fsi.replace("  elPropId = 1\n", "  elPropId = 1\n  alpha1 = 0.5\n  alpha2 = 3.0e-4\n")
    return fsi


def _cases():
    dyn = ["-timeInc=0.001", "-timeEnd=0.005", "-alphaNewmark=0.1", "-tolDispNorm=1.0e-8"]
    qs = ["-timeInc=0.01", "-timeEnd=0.06", "-quasiStatic=0.03", "-tolDispNorm=1.0e-9"]
    return [(_chain(20, damped=True), dyn), (_chain(47, damped=True), dyn), (_chain(20), qs),
            (_chain(16, motion=(16, 2, 0.2)), ["-numit=-1"] + qs), (_chain(20, damped=True), qs)]


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_alone_and_beside_long_chains_agree_bitwise(gpu, mixed):
    from fedem_gb300 import models
    from fedem_gb300.batch import Batch, create_models

    cases = _cases()
    big = [models.batch_c4(1, seed=s, n_min=30000, n_max=30000, steps=4)[0][:2] for s in range(6)]
    ms = create_models(cases + big)
    together = Batch(ms, mixed=mixed)
    assert together.run()["models_failed"] == 0
    for k in range(len(cases)):
        alone = Batch([ms[k]], mixed=mixed)
        assert alone.run()["models_failed"] == 0
        np.testing.assert_array_equal(together.triads(k), alone.triads(0))
        np.testing.assert_array_equal(together.norms(k), alone.norms(0))
        assert together.info(k)["iterations"] == alone.info(0)["iterations"]
        alone.close()
    together.close()
