"""The large-front launches are cooperative: all blocks are resident, so there may be no
more of them than the device, or the partition of it that the process has, holds.  Frames
planned for fewer SMs than the device has (FGPU_LARGE_SMS at batch creation) must launch
at most so many blocks, or four times as many where most levels have more fronts than SMs,
and give the same bits: every entry's arithmetic is the same whichever block does it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("sms", [1, 3, 20, 75])
def test_fewer_blocks_same_bits(gpu, monkeypatch, sms, mixed):
    from fedem_gb300 import models
    from fedem_gb300.batch import Batch, Model

    ms = [Model(*models.space_frame_c2(seed=11, storeys=s, bays=b, n_joints=2, n_springs=2, steps=3))
          for s, b in ((3, 1), (4, 2), (3, 3))]
    whole = Batch(ms, mixed=mixed)
    monkeypatch.setenv("FGPU_LARGE_SMS", str(sms))
    part = Batch(ms, mixed=mixed)
    assert part.front_plan()["large"] == whole.front_plan()["large"] > 0
    assert 0 < part.front_plan()["large_blocks"] <= 4 * sms
    if sms >= 20:  # no level of three frames has so many fronts
        assert part.front_plan()["large_blocks"] <= sms
    for b in (whole, part):
        assert b.run()["models_failed"] == 0
    for k in range(len(ms)):
        np.testing.assert_array_equal(part.triads(k), whole.triads(k))
        np.testing.assert_array_equal(part.norms(k), whole.norms(k))
    whole.close()
    part.close()


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_many_models_several_blocks_per_sm(gpu, tmp_path, mixed):
    """Batches whose levels have more large fronts than the GPU has SMs run several blocks
    per SM, on kernels of their own register count; a model alone does not (bitwise)."""
    import torch
    from fedem_gb300 import models
    from fedem_gb300.batch import Batch, Model

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for m in (Model(*models.superelement_chain_c3(str(tmp_path), n_parts=6, n_modes=36, steps=3)[:2]),
              Model(*models.space_frame_c2(seed=21, storeys=3, bays=2, n_joints=2, n_springs=2, steps=3))):
        many, alone = Batch([m] * (2 * sms), mixed=mixed), Batch([m], mixed=mixed)
        assert alone.front_plan()["large_blocks"] <= sms < many.front_plan()["large_blocks"]
        for b in (many, alone):
            assert b.run()["models_failed"] == 0
        for k in (0, 1, sms, 2 * sms - 1):
            np.testing.assert_array_equal(many.triads(k), alone.triads(0))
            np.testing.assert_array_equal(many.norms(k), alone.norms(0))
        many.close()
        alone.close()
