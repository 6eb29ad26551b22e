"""The power-of-two register and TMA-fed passes on problems small enough for the oracle.

Plans take them by themselves only above 2^19 cells (3-D; 2-D grids by their size), so
the cases of the physics, field, golden and adjoint tests run here once more with the
mixed-radix passes off (KWAVE_GB300_MR=0, read when a plan is finalized), each against
the same oracle and with the same bounds as there.  The geometry tuner runs on a plan
that its kernels serve, and has to time its candidates.
"""
import ctypes as C

import numpy as np
import pytest

import test_adjoint_gpu as adjoint
import test_fields_gpu as fields
import test_parity_gpu as parity
import test_physics_gpu as physics

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def no_mixed_radix(monkeypatch):
    monkeypatch.setenv("KWAVE_GB300_MR", "0")


@pytest.mark.parametrize("kind,shape", physics.CASES, ids=[f"{k}-{'x'.join(map(str, s))}" for k, s in physics.CASES])
def test_physics(kind, shape):
    physics.test_power_of_two_physics(kind, shape)


@pytest.mark.parametrize("shape", [s for s in fields.SHAPES if any(n >= 64 for n in s)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("pml", [0, 2])
def test_fields(shape, pml):
    fields.test_state_after_each_step(shape, pml)


@pytest.mark.parametrize("name", parity.case_names())
def test_golden(name):
    parity.test_gpu_matches_reference(name)


@pytest.mark.parametrize("name", sorted(adjoint.CASES))
def test_adjoint(name):
    adjoint.test_adjoint_matches_oracle(name)


@pytest.mark.parametrize("name", sorted(adjoint.C_CASES))
def test_sound_speed_gradient(name):
    adjoint.test_sound_speed_gradient_matches_oracle(name)


def test_cartesian_circle_adjoint():
    adjoint.test_cartesian_circle_adjoint_128()


# k-space corrected velocity sources, velocities recorded on the pressure grid and a
# recording that starts late, beside every kind of medium, on power-of-two 3-D rows
@pytest.mark.parametrize("medium", ["lossless", "nonlinear", "stokes", "powerlaw"])
@pytest.mark.parametrize("shape", [(64, 20, 128), (16, 64, 256), (128, 128)], ids=lambda s: "x".join(map(str, s)))
def test_sources_and_velocity_records(shape, medium):
    from kwave_gb300.solver import Simulation
    from oracle.kspace_oracle import OracleSimulation

    rng = np.random.default_rng(sum(shape))
    mask = rng.random(shape) < 0.02
    mask.flat[0] = mask.flat[-1] = True
    n = int(mask.sum())
    prob = dict(shape=shape, spacing=(1e-4,) * len(shape), dt=1.5e-8, Nt=6,
                sound_speed=1500.0 * (1 + 0.05 * rng.standard_normal(shape)),
                density=1000.0 * (1 + 0.05 * rng.standard_normal(shape)), u_mask=mask,
                ux=1e-6 * rng.standard_normal((n, 6)), uy=1e-6 * rng.standard_normal((1, 4)), u_mode="additive",
                p_mask=mask, p=rng.standard_normal((n, 3)), p_mode="additive", sensor_mask=np.ones(shape, bool),
                record=("p", "u"), record_start_index=3, pml_size=(2,) * len(shape), pml_alpha=(2.0,) * len(shape),
                use_sg=True, use_kspace=True, smooth_p0=False)
    if medium == "nonlinear":
        prob["BonA"] = 6.0
    elif medium != "lossless":
        prob.update(alpha_coeff=0.75, alpha_power=2.0 if medium == "stokes" else 1.5)
    ref = OracleSimulation(prob, np.float64).setup()
    want = ref.run()
    sim = Simulation.from_problem(prob)
    try:
        got = sim.run()
        got.update({"field_p": sim.p}, **{f"field_u{i}": f for i, f in enumerate(sim.u)})
    finally:
        sim.close()
    want.update({"field_p": ref.p}, **{f"field_u{i}": f for i, f in enumerate(ref.u)})
    for k, v in want.items():
        err = np.linalg.norm(got[k] - v) / np.linalg.norm(v)
        # relative L2 of float32 transforms, as tests/test_mixed_radix_gpu.py asks over four steps
        assert err <= 2e-6, (k, err)


def test_autotune_times_its_candidates():
    import bench
    from kwave_gb300 import _lib
    from kwave_gb300.solver import Simulation

    prob = bench.transmit_problem((90, 150), 11, nt=40, n_elem=6, pml=12)

    def launches(sim):
        n = C.c_int64()
        _lib.check(_lib.lib().kw_plan_launch_count(sim._plan.handle, C.byref(n)))
        return n.value

    sim = Simulation.from_problem(prob)
    sim.setup()
    try:
        ref = sim.run()
        per_step = launches(sim) / sim.Nt
    finally:
        sim.close()
    sim = Simulation.from_problem(prob)
    sim.setup(autotune=True)
    try:
        # four tile widths x three numbers of rows, each over at least four steps
        assert launches(sim) >= 12 * 4 * 0.5 * per_step
        assert sim._plan.time_index() == 0
        got = sim.run()
        for k, v in ref.items():
            assert np.array_equal(v, got[k]), k
    finally:
        sim.close()
