"""Which passes 2-D grids take whose rows are longer than the mixed-radix row kernels
allow (1024 complex points): columns of 64, 128, 256 and 1024 points stay on the
power-of-two passes, which are faster there, so that the whole step is what
KWAVE_GB300_MR=0 gives, bit for bit; 512 and other lengths are on the mixed-radix
passes, within the float32 rounding of the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,same", [((64, 2058), True), ((128, 1029), True), ((256, 2187), True), ((1024, 2100), True),
                                        ((512, 2058), False), ((96, 1029), False), ((256, 2048), False)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else None)
def test_route(shape, same, monkeypatch):
    from kwave_gb300.solver import Simulation

    rng = np.random.default_rng(shape[1])
    prob = dict(shape=shape, spacing=(1e-4, 1e-4), dt=1.5e-8, Nt=4, density=1000.0, p0=rng.standard_normal(shape),
                sound_speed=1500.0 * (1 + 0.02 * rng.standard_normal(shape)), alpha_coeff=0.75, alpha_power=1.5, BonA=6.0,
                smooth_p0=False, sensor_mask=None, record=("p",), pml_size=(4, 4), pml_alpha=(2.0, 2.0))

    def run():
        sim = Simulation.from_problem(prob)
        try:
            sim.run()
            return [sim.p, *sim.u, *sim.rho_split]
        finally:
            sim.close()

    got = run()
    monkeypatch.setenv("KWAVE_GB300_MR", "0")
    want = run()
    assert all(np.array_equal(a, b) for a, b in zip(got, want)) == same
    for a, b in zip(got, want):
        assert np.linalg.norm(a - b) <= 4e-6 * np.linalg.norm(b)  # twice the bound against the oracle
