"""Served engines of models with large fronts: the large fronts' launches take the whole
GPU with all blocks resident, so those of engines that run at the same time follow one
another; frames and part chains, two to an engine and several engines at once, give the
bits of the model alone."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_engines_of_frames_and_parts(gpu, tmp_path, mixed):
    from fedem_gb300 import models
    from fedem_gb300.batch import Batch, Model, Server

    cases = [models.space_frame_c2(seed=20 + k, storeys=4 + k, bays=2, n_joints=2, n_springs=2, steps=12)
             for k in range(4)]
    cases += [models.superelement_chain_c3(str(tmp_path), n_parts=p, n_modes=30, steps=12)[:2] for p in (4, 6)]
    ms = [Model(*c[:2]) for c in cases]
    srv = Server(budget_bytes=8e9, mixed=mixed, max_models_per_batch=2, min_batch=1, max_wait=0.0)
    srv.set_max_engines(3)
    ids = [srv.submit(m) for m in ms]
    t0, live = time.time(), 0
    while any(srv.request(i)["state"] < 2 for i in ids):
        srv.pump()
        live = max(live, srv.status()["live_batches"])
        assert time.time() - t0 < 120
    assert live >= 2
    for m, i in zip(ms, ids):
        r = srv.request(i)
        assert r["state"] == 2, r
        alone = Batch([m], mixed=mixed)
        alone.run()
        np.testing.assert_array_equal(srv.result(i), alone.triads(0))
        assert r["iterations"] == alone.info(0)["iterations"]
        alone.close()
    srv.close()
