"""A kernel launch that the runtime refuses (made by the host: the hook asks for more
shared memory than any device has) must fail the call that made it, whichever of the
call's launches it is, and leave nothing behind: no result of an earlier call reported as
the new one, no captured iteration with a kernel missing, no error in another batch's
call.  Done again, the call gives the same bits as one that nothing disturbed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPTS = ["-timeInc=0.001", "-timeEnd=0.006", "-alphaNewmark=0.1", "-tolDispNorm=1.0e-10"]


def _chain():
    from fedem_gb300 import models

    return models.beam_chain_fsi(30, 0.25, 0.1, 0.01, clamp=0, load_node=30, load_dof=2, load=1200.0,
                                 **models.STEEL), OPTS


def _frame():
    from fedem_gb300 import models

    return models.space_frame_c2(seed=11, storeys=3, bays=2, n_joints=2, n_springs=2, steps=3)


CASES = [(_chain, False), (_chain, True), (_frame, False), (_frame, True)]
IDS = ["chain_fp64", "chain_mixed", "frame_fp64", "frame_mixed"]


def _each_launch(lib, call, check):
    """call() with its 1st, 2nd, ... launch refused, up to the last; check() after each."""
    from fedem_gb300 import FedemException

    refused = 0
    for n in range(1, 1000):
        lib.fgpu_probe_refuse_launch(n)
        try:
            call()
            failed = False
        except FedemException:
            failed = True
        if lib.fgpu_probe_refuse_launch(0) > 0:  # fewer launches than n
            assert not failed
            break
        refused += 1
        assert failed, f"launch {n} was refused, the call reported success"
        check()
    assert refused > 0
    return refused


@pytest.mark.parametrize("make,mixed", CASES, ids=IDS)
def test_seam(gpu, make, mixed):
    from fedem_gb300 import load_library
    from fedem_gb300.batch import Batch, Model

    lib = load_library()
    m = Model(*make())
    b = Batch([m], mixed=mixed)
    rhs = np.random.default_rng(3).standard_normal((2, m.neq))

    def solve():
        b.assemble_newton(0, 3.0e6, 0.0, 0.9)
        assert b.factor(0) == 0
        return b.solve(0, rhs)

    want = solve()
    for call in (lambda: b.assemble_newton(0, 4.0e6, 0.0, 0.9), lambda: b.factor(0), lambda: b.solve(0, 2.0 * rhs)):
        _each_launch(lib, call, lambda: np.testing.assert_array_equal(solve(), want))
    b.close()
    m.close()


@pytest.mark.parametrize("make,mixed", CASES, ids=IDS)
def test_run(gpu, make, mixed):
    """(with the launch shapes fixed: refused launches of the autotuner's probe fail only
    the probe, see below)"""
    from fedem_gb300 import FedemException, load_library
    from fedem_gb300.batch import Batch, Model

    lib = load_library()
    m = Model(*make())
    ref = Batch([m], mixed=mixed)
    ref.set_launch_shape(0, 8, 8, 16)
    assert ref.run()["models_done"] == 1
    b = Batch([m], mixed=mixed)
    b.set_launch_shape(0, 8, 8, 16)
    b.snapshot()

    def again():
        b.restore()
        assert b.run()["models_done"] == 1
        np.testing.assert_array_equal(b.triads(0), ref.triads(0))
        b.restore()

    # the first captures the iteration, and no graph may be kept with a kernel missing
    lib.fgpu_probe_refuse_launch(3)
    with pytest.raises(FedemException):
        b.run()
    assert lib.fgpu_probe_refuse_launch(0) == 0
    again()
    # the launches of a run whose iterations are captured already: the last step start
    _each_launch(lib, b.run, again)
    ref.close()
    b.close()
    m.close()


@pytest.mark.parametrize("make,mixed", CASES, ids=IDS)
def test_create_and_first_run(gpu, make, mixed):
    """Every launch from the batch's creation on: the initial state, the autotuner's probe
    (which then keeps the default shapes) and both captured iterations."""
    from fedem_gb300 import FedemException, load_library
    from fedem_gb300.batch import Batch, Model

    lib = load_library()
    m = Model(*make())
    ref = Batch([m], mixed=mixed)
    assert ref.run()["models_done"] == 1
    want = ref.triads(0).copy()
    ref.close()
    for n in [*range(1, 40), *range(40, 400, 7)]:
        lib.fgpu_probe_refuse_launch(n)
        b = None
        try:
            b = Batch([m], mixed=mixed)
            b.run()
            failed = False
        except FedemException:
            failed = True
        left = lib.fgpu_probe_refuse_launch(0)
        if b is not None:
            if failed:
                b.run()  # goes on from where the refused call stopped
            assert b.info(0)["state"] == 2
            np.testing.assert_array_equal(b.triads(0), want)
            b.close()
        if left > 0:
            break
    m.close()


def test_externally_driven_step(gpu):
    from fedem_gb300 import load_library
    from fedem_gb300.solver import FedemSolver

    lib = load_library()
    fsi, opts = _chain()
    s = FedemSolver(solver_options=opts, fsi=fsi)
    assert s.solve_next() and s.ierr.value == 0
    assert s.start_step()
    for n in (1, 5):
        lib.fgpu_probe_refuse_launch(n)
        assert not s.finish_step()
        assert lib.fgpu_probe_refuse_launch(0) == 0
        assert s.ierr.value < 0
        s.solver_done()
        s = FedemSolver(solver_options=opts, fsi=fsi)
        assert s.start_step()
    s.solver_done()
