"""Mixed-radix row stages and axis passes (csrc/kw_mr*.cu*) at the sizes where
they can go wrong: the smallest and largest lengths, two, three and four
passes, padded and unpadded last radices, odd rows (two to a transform, with
and without a row left over), blocks that end inside the grid, and lengths on
either side of the limits where other kernels take over.

Every field after four steps, and the recorded velocity on the pressure grid,
against the oracle in float64: relative L2 at most 2e-6 (four steps of
float32 transforms, each within a few 1e-7), as tests/test_fields_gpu.py asks
of the other kernels.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    (4, 8),            # two radix-2 passes along both axes
    (9, 15),           # odd rows, one left over
    (10, 14),          # rows of 7 pairs: a prime, generic rows beside mixed-radix columns
    (15, 25),
    (21, 48),
    (49, 30),
    (343, 20),         # three passes of 7
    (16, 1250),        # four passes of 5 along rows
    (625, 18),         # four passes of 5 along columns
    (12, 2048),        # 1024 pairs, the most a row block takes
    (10, 2058),        # 1029 pairs, one size on: generic rows
    (6, 945),          # long odd rows
    (2401, 10),        # four passes of 7, the longest column of that kind
    (6, 10, 9),        # 3-D, odd rows and an odd number of them
    (9, 15, 27),
    (12, 7, 20),       # a prime axis: generic passes along y
    (24, 18, 40),
    (32, 64, 36),      # power-of-two columns beside mixed-radix rows
]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("medium", ["lossless", "stokes", "powerlaw"])
def test_fields_vs_oracle(shape, medium):
    from kwave_gb300.solver import Simulation
    from oracle.kspace_oracle import OracleSimulation

    rng = np.random.default_rng(sum(shape))
    c = 1500.0 * (1 + 0.05 * rng.standard_normal(shape))
    prob = dict(shape=shape, spacing=(1e-4,) * len(shape), dt=1.5e-8, Nt=4, sound_speed=c,
                density=1000.0 * (1 + 0.05 * rng.standard_normal(shape)), p0=rng.standard_normal(shape), smooth_p0=False,
                sensor_mask=np.ones(shape, bool), record=("p", "u"), pml_size=(2,) * len(shape),
                pml_alpha=(2.0,) * len(shape), use_sg=True, use_kspace=True)
    if medium != "lossless":
        prob.update(alpha_coeff=0.75, alpha_power=2.0 if medium == "stokes" else 1.5, BonA=6.0)
    if medium == "powerlaw":  # and sources: k-space corrected pressure, sparse velocity
        mask = rng.random(shape) < 0.1
        mask.flat[0] = True
        prob.update(p_mask=mask, p=rng.standard_normal((int(mask.sum()), 3)), p_mode="additive",
                    u_mask=mask, ux=1e-7 * rng.standard_normal((int(mask.sum()), 4)), u_mode="additive-no-correction")
    if medium == "stokes":  # sparse pressure, k-space corrected velocity
        mask = rng.random(shape) < 0.1
        mask.flat[-1] = True
        prob.update(p_mask=mask, p=rng.standard_normal((1, 3)), p_mode="additive-no-correction",
                    u_mask=mask, uy=1e-7 * rng.standard_normal((int(mask.sum()), 4)), u_mode="additive")
    ref = OracleSimulation(prob, np.float64).setup()
    want = ref.run()
    sim = Simulation.from_problem(prob)
    try:
        got = sim.run()
        got.update({"field_p": sim.p}, **{f"field_u{i}": f for i, f in enumerate(sim.u)},
                   **{f"field_rho{i}": f for i, f in enumerate(sim.rho_split)})
    finally:
        sim.close()
    want.update({"field_p": ref.p}, **{f"field_u{i}": f for i, f in enumerate(ref.u)},
                **{f"field_rho{i}": f for i, f in enumerate(ref.rho_split)})
    for k, v in want.items():
        err = np.linalg.norm(got[k] - v) / np.linalg.norm(v)
        assert err <= 2e-6, (k, err)


def test_batch_sources_end_at_different_steps():
    """Grouped launches hold the source passes until the last member's k-space
    corrected source ends; members of every parity and dimension, with
    pressure or velocity sources or none, equal their solo runs bit for bit."""
    from kwave_gb300.solver import run_problem, SimulationBatch

    probs = []
    for i, (shape, length) in enumerate([((48, 60), 12), ((45, 75), 40), ((64, 128), 25), ((20, 18, 24), 33),
                                         ((15, 21, 25), 18), ((50, 54), 0)]):
        rng = np.random.default_rng(i)
        mask = np.zeros(shape, bool)
        mask.flat[rng.choice(mask.size, 9, replace=False)] = True
        p = dict(shape=shape, spacing=(1e-4,) * len(shape), dt=1.5e-8, Nt=60,
                 sound_speed=1500.0 * (1 + 0.02 * rng.standard_normal(shape)), density=1000.0, alpha_coeff=0.5,
                 alpha_power=1.1, sensor_mask=rng.random(shape) < 0.05, record=("p", "ux"), pml_size=(4,) * len(shape),
                 pml_alpha=(2.0,) * len(shape), use_sg=True, use_kspace=True, smooth_p0=False)
        if length == 0:
            p["p0"] = rng.standard_normal(shape)
        elif i % 2:
            p.update(u_mask=mask, ux=1e-6 * rng.standard_normal((9, length)), u_mode="additive")
        else:
            p.update(p_mask=mask, p=rng.standard_normal((9, length)), p_mode="additive")
        probs.append(p)
    solo = [run_problem(p) for p in probs]
    batch = SimulationBatch.from_problems(probs)
    try:
        got = batch.run()
    finally:
        batch.close()
    for i, (a, b) in enumerate(zip(got, solo)):
        for k in b:
            assert np.array_equal(a[k], b[k]), (i, k)
