"""A batch member in the wait test (kw_plan_set_wait_test) on a grid of the mixed-radix
passes: its velocity stage runs on the bulk-fed kernel, so it is not grouped with the
others; the withheld copy's wait runs out, the batch reports it, and the device stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_timeout_in_a_batch():
    from kwave_gb300 import _lib
    from kwave_gb300.solver import Simulation, SimulationBatch, run_problem

    def problem(shape):
        p0 = np.zeros(shape)
        p0[shape[0] // 2, shape[1] // 2] = 1.0
        return dict(shape=shape, spacing=(1e-4, 1e-4), dt=2e-8, Nt=9, sound_speed=1500.0, density=1000.0, p0=p0,
                    smooth_p0=False, sensor_mask=p0 == 0, record=("p",), pml_size=(8, 8), pml_alpha=(2.0, 2.0))

    probs = [problem((64, 128)), problem((60, 72))]
    sims = [Simulation.from_problem(p).setup() for p in probs]
    _lib.check(_lib.lib().kw_plan_set_wait_test(sims[0]._plan.handle, 1))
    batch = SimulationBatch(sims)
    try:
        batch.run_steps(6)
        with pytest.raises(_lib.KwaveGB300Error, match="timed out"):
            sims[0]._plan.sync()
    finally:
        batch.close()
    batch = SimulationBatch.from_problems(probs)
    try:
        for p, got in zip(probs, batch.run()):
            assert np.array_equal(got["p"], run_problem(p)["p"])
    finally:
        batch.close()
