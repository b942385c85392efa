"""Several batches in one process.  Kernels whose blocks need more than 48 KB of shared
memory get a limit that is an attribute of the function, not of a launch: a batch must
run the same whichever other batches were created, or step on another host thread, in
between (bitwise, tolerance zero)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_parts_of_another_size_created_in_between(gpu, tmp_path):
    """Parts of 72 DOFs (83 KB for the Newton matrix of one) run after a batch of parts of
    18 DOFs was created, against the run before it."""
    from fedem_gb300 import models
    from fedem_gb300.batch import Batch, Model

    def part_chain(n_modes):
        d = tmp_path / str(n_modes)
        d.mkdir()
        return Model(*models.superelement_chain_c3(str(d), n_parts=2, n_modes=n_modes, steps=5)[:2])

    big, small = part_chain(60), part_chain(6)
    alone = Batch([big])
    assert alone.run()["models_failed"] == 0
    b = Batch([big])
    other = Batch([small])
    assert b.run()["models_failed"] == 0, b.info(0)
    assert other.run()["models_failed"] == 0
    np.testing.assert_array_equal(b.triads(0), alone.triads(0))
    for x in (alone, b, other):
        x.close()


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_two_threads_solve_with_fronts_of_different_sizes(gpu, mixed):
    """A frame's small fronts (up to 48 rows) and a chain's (30 rows) take different amounts
    of shared memory in the same kernels: two threads factor and solve at once, each with
    right-hand sides in turn, and get the solutions of one thread alone."""
    from fedem_gb300 import models
    from fedem_gb300.batch import Batch, Model

    cases = [models.space_frame_c2(seed=11, storeys=6, bays=2, n_joints=2, n_springs=2, steps=3),
             models.batch_c4(1, seed=7, n_min=400, n_max=400, steps=3)[0][:2]]
    ms = [Model(*c) for c in cases]
    bs = [Batch([m], mixed=mixed) for m in ms]
    rng = np.random.default_rng(5)
    rhs = [rng.standard_normal((5, m.neq)) for m in ms]
    want, scales = [], (3.0e6, 4.0e6, 5.0e6)
    for b, r in zip(bs, rhs):
        per = []
        for s in scales:
            b.assemble_newton(0, s, 0.0, 0.9)
            assert b.factor(0) == 0
            per.append([b.solve(0, r[k:k + 1]) for k in range(5)])
        want.append(per)
    wrong = [0, 0]

    def work(i):
        for n in range(60):
            j = n % len(scales)
            bs[i].assemble_newton(0, scales[j], 0.0, 0.9)
            if bs[i].factor(0) != 0:
                wrong[i] += 1
            for k in range(5):
                wrong[i] += not np.array_equal(bs[i].solve(0, rhs[i][k:k + 1]), want[i][j][k])

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [0, 0]
    for b in bs:
        b.close()
