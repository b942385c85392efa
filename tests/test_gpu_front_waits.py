"""The bounded waits of the trees on thread blocks and of the large-front kernels, each made
to run out on the probe's own counters (nothing faults, traps or hangs): the wait sets the
batch's error flag, a kernel that goes on runs to its end, the running models fail with
SS_TIMEOUT, and the context stays usable: a new batch gives the bits of one before."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ST_ERROR, SS_TIMEOUT = 3, 16


def _model(kind):
    from fedem_gb300 import models
    from fedem_gb300.batch import Model

    if kind == "chain":
        return Model(*models.batch_c4(1, seed=5, n_min=120, n_max=120, steps=4)[0][:2])
    return Model(*models.space_frame_c2(seed=11, storeys=4, bays=2, n_joints=2, n_springs=2, steps=3))


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("kind,which", [("chain", 0), ("chain", 1), ("frame", 2), ("frame", 3)],
                         ids=["tree_slot", "tree_root", "large_children", "large_blocks"])
def test_wait_runs_out_and_fails_the_models(gpu, kind, which, mixed):
    from fedem_gb300 import load_library
    from fedem_gb300.batch import Batch

    lib = load_library()
    m = _model(kind)
    ref = Batch([m], mixed=mixed)
    plan = ref.front_plan()
    assert plan["tree_warps" if kind == "chain" else "large"] > 0
    assert ref.run()["models_done"] == 1
    b = Batch([m], mixed=mixed)
    flag = ctypes.c_int(0)
    assert lib.fgpu_batch_probe_front_wait_timeout(b._h, which, 4096, ctypes.byref(flag)) == 0, lib.fgpu_last_error()
    assert flag.value == 1
    b.run()
    info = b.info(0)
    assert info["state"] == ST_ERROR and (info["status"] & SS_TIMEOUT)
    b.close()
    b2 = Batch([m], mixed=mixed)
    assert b2.run()["models_done"] == 1
    np.testing.assert_array_equal(b2.triads(0), ref.triads(0))
    for x in (b2, ref):
        x.close()
    m.close()


def test_probe_without_such_fronts_is_refused(gpu):
    from fedem_gb300 import load_library
    from fedem_gb300.batch import Batch

    lib = load_library()
    b = Batch([_model("chain")])
    flag = ctypes.c_int(0)
    for which in (-1, 2, 3, 4):
        assert lib.fgpu_batch_probe_front_wait_timeout(b._h, which, 4096, ctypes.byref(flag)) != 0
    b.close()
