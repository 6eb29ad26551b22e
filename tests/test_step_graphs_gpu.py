"""Graphs of several steps, and passes launched as programmatic dependents: a run
cut into pieces of any length, a run of plain launches and one run give the same
bits, with sources that end and a recording that begins inside a graph's span."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _prob(shape):
    rng = np.random.default_rng(len(shape))
    mask = rng.random(shape) < 0.02
    mask.flat[0] = True
    return dict(shape=shape, spacing=(1e-4,) * len(shape), dt=1.5e-8, Nt=131,
                sound_speed=1500.0 * (1 + 0.05 * rng.standard_normal(shape)), density=1000.0, alpha_coeff=0.75,
                alpha_power=1.5, BonA=6.0, p0=rng.standard_normal(shape), smooth_p0=False,
                p_mask=mask, p=rng.standard_normal((int(mask.sum()), 53)), p_mode="additive",
                u_mask=mask, ux=1e-7 * rng.standard_normal((int(mask.sum()), 90)), u_mode="additive-no-correction",
                sensor_mask=np.ones(shape, bool), record=("p", "u"), record_start_index=21,
                pml_size=(2,) * len(shape), pml_alpha=(2.0,) * len(shape), use_sg=True, use_kspace=True)


@pytest.mark.parametrize("shape", [(30, 28), (20, 18, 15), (32, 32, 64)], ids=lambda s: "x".join(map(str, s)))
def test_pieces_and_plain_launches(shape, monkeypatch):
    from kwave_gb300.solver import Simulation

    def run(pieces):
        sim = Simulation.from_problem(_prob(shape))
        try:
            sim.setup()
            for n in pieces:
                sim._plan.run(n)
            sim.t = sim._plan.time_index()
            out = sim.run()
            out["field_p"] = sim.p
            return out
        finally:
            sim.close()

    whole = run([])
    assert whole["p"].shape[-1] == 131 - 20 and np.isfinite(whole["p"]).all() and np.abs(whole["p"]).max() > 0
    cut = run([1, 41, 8, 33, 9])
    monkeypatch.setenv("KWAVE_GB300_GRAPHS", "0")
    plain = run([])
    for k, v in whole.items():
        assert np.array_equal(v, cut[k]) and np.array_equal(v, plain[k]), k
