"""Phase timings: of a run of limited length every seventh iteration is sampled, and the
last one, so that a run of fewer than seven has a sample too."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 6, 7, 8, 13, 14, 20])
def test_samples_of_a_limited_run(gpu, n):
    from fedem_gb300 import models
    from fedem_gb300.batch import Batch, Model

    fsi, opts = models.cantilever_c1()
    m = Model(fsi, opts)
    b = Batch([m])
    b.phase_timings(reset=True)
    assert b.run(max_batched=n)["batched_iterations"] == n
    samples, ms, elements = b.phase_timings(reset=True)
    assert samples == n // 7 + (n % 7 > 0)
    assert elements == samples * m.nel and all(t > 0 for t in ms[:3])
    b.close()
