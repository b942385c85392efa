"""Which kernels take the small fronts: trees on thread blocks where their chunks are few
or well filled (all small fronts, 16 or 8 warps a block, or only the upper levels), else
the cascades; a chunk is of one model, so a batch of many small models belongs to the
cascades.  Every tier gives the bits of the model alone (tolerance zero)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# models, beams each, warps per chunk (0: cascades), the trees take all small fronts
CASES = [(1, 20, 16, True), (100, 8, 16, True), (64, 150, 16, True), (300, 40, 8, True), (5, 4000, 16, False),
         (4000, 1, 0, False), (1000, 3, 0, False), (1000, 8, 0, False), (300, 12, 0, False)]


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n_models,n_el,warps,whole", CASES)
def test_plan_and_bits(gpu, n_models, n_el, warps, whole, mixed):
    from fedem_gb300 import models
    from fedem_gb300.batch import Batch, create_models

    ms = create_models([c[:2] for c in models.batch_c4(n_models, seed=3, n_min=n_el, n_max=n_el, steps=3)])
    b = Batch(ms, mixed=mixed)
    plan = b.front_plan()
    assert plan["tree_warps"] == warps and (plan["tree_chunks"] > 0) == (warps > 0)
    if warps:  # all: a leaf chunk per 16 or 8 fronts at least; upper levels: far fewer
        assert (plan["tree_chunks"] * warps >= plan["fronts"]) == whole
    assert b.run()["models_failed"] == 0
    for k in sorted({0, n_models // 2, n_models - 1}):
        alone = Batch([ms[k]], mixed=mixed)
        assert alone.run()["models_failed"] == 0
        np.testing.assert_array_equal(b.triads(k), alone.triads(0))
        np.testing.assert_array_equal(b.norms(k), alone.norms(0))
        alone.close()
    b.close()
