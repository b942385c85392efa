"""Small batches take kernels of their own: four lanes per beam element in the
element pass and the Newton matrices (up to 8,192 elements), clusters of one-warp
blocks in the norms (up to 48 chunks), four lanes per joint, and the assembly trees on
thread blocks (up to 8,192 leaf fronts; up to 32,768 the trees' upper levels only,
their many backward roots seeded by sixteen warps).  They perform the operations of
the large batches' kernels in the same order, so a model alone and the same model
beside two long chains (the trees' upper levels) or six (the cascades alone), which
put the batch above the other lines, must agree to the last bit (tolerance zero):
chains from a single beam (one front) over the sizes around the chunks' tiers, and a
gravity-loaded pendulum with a joint (kept frames, gravity forces, constraint
expansion)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPTS = ["-timeInc=0.001", "-timeEnd=0.004", "-alphaNewmark=0.1", "-tolDispNorm=1.0e-8"]


def _cases():
    from fedem_gb300 import models

    out = [models.batch_c4(1, seed=60 + n, n_min=n, n_max=n, steps=4)[0][:2] for n in (1, 2, 3, 4, 9, 47, 95, 400)]
    out.append((models.pendulum(n_el=6)[0], OPTS))
    return out


@pytest.mark.parametrize("chains", [2, 6])
@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_alone_and_in_a_large_batch_agree_bitwise(gpu, mixed, chains):
    from fedem_gb300 import models
    from fedem_gb300.batch import Batch, create_models

    cases = _cases()
    big = [models.batch_c4(1, seed=s, n_min=30000, n_max=30000, steps=4)[0][:2] for s in range(chains)]
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


def test_many_joints_agree_bitwise_with_one(gpu):
    """Beyond 4,864 joints a joint has one lane; 4,900 pendulums against one alone (the
    joint's four lanes, and every other small-batch kernel)."""
    from fedem_gb300 import models
    from fedem_gb300.batch import Batch, Model

    m = Model(models.pendulum(n_el=2)[0], OPTS)
    alone, many = Batch([m]), Batch([m] * 4900)
    assert alone.run()["models_failed"] == 0 and many.run()["models_failed"] == 0
    for k in (0, 1, 2500, 4899):
        np.testing.assert_array_equal(many.triads(k), alone.triads(0))
        np.testing.assert_array_equal(many.norms(k), alone.norms(0))
    alone.close()
    many.close()
