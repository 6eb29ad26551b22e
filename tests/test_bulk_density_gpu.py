"""The bulk-fed density stage of linear media without power-law absorption
(k_rows_tma, ST_RHO) against the register row kernel it takes the place of: the same
operations in the same order, so the same bits.  Row lengths of every transform size,
a last block of rows that is not full, scalar and grid media, Stokes absorption, a
sparse pressure source and a last step that writes p."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 3, 128), (8, 8, 256), (4, 3, 512), (3, 4, 1024), (2, 3, 2048), (6, 256), (128, 96, 128)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("medium", ["scalar", "grid", "stokes"])
def test_same_bits_as_register_kernel(shape, medium, monkeypatch):
    from kwave_gb300.solver import Simulation

    rng = np.random.default_rng(sum(shape))
    grid = (lambda m, s: m * (1 + s * rng.standard_normal(shape))) if medium != "scalar" else (lambda m, s: m)
    mask = rng.random(shape) < 0.05
    mask.flat[0] = mask.flat[-1] = True
    prob = dict(shape=shape, spacing=(1e-4,) * len(shape), dt=1.5e-8, Nt=5, sound_speed=grid(1500.0, 0.05),
                density=grid(1000.0, 0.05), p0=rng.standard_normal(shape), smooth_p0=False,
                p_mask=mask, p=rng.standard_normal((1, 4)), p_mode="additive-no-correction",
                sensor_mask=np.ones(shape, bool), record=("p",), pml_size=(1,) * len(shape),
                pml_alpha=(2.0,) * len(shape), use_sg=True, use_kspace=True)
    if medium == "stokes":
        prob.update(alpha_coeff=grid(0.75, 0.1), alpha_power=2.0)

    def run():
        sim = Simulation.from_problem(prob)
        try:
            out = sim.run()
            out.update({"field_p": sim.p}, **{f"rho{i}": f for i, f in enumerate(sim.rho_split)})
            return out
        finally:
            sim.close()

    monkeypatch.setenv("KWAVE_GB300_MR", "0")
    bulk = run()
    monkeypatch.setenv("KWAVE_GB300_ROWS_TMA", "0")
    reg = run()
    assert np.abs(bulk["p"]).max() > 0
    for k, v in reg.items():
        assert np.array_equal(v, bulk[k]), k
