"""Members of a 3-D batch whose k-space corrected source is over before another
member's: none of their source passes works any more, so the source spectra stay what
the last step with a source left, as in a run alone.  (With the y passes left on they
grew by N_y a step, to infinity.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(i, shape, kind, length):
    rng = np.random.default_rng(i)
    mask = np.zeros(shape, bool)
    mask.flat[rng.choice(mask.size, 7, replace=False)] = True
    p = dict(shape=shape, spacing=(1e-4,) * 3, dt=1.5e-8, Nt=60, sound_speed=1500.0, density=1000.0,
             sensor_mask=rng.random(shape) < 0.05, record=("p",), pml_size=(2,) * 3, pml_alpha=(2.0,) * 3, use_sg=True,
             use_kspace=True, smooth_p0=False)
    signal = rng.standard_normal((7, length))
    return dict(p, p_mask=mask, p=signal, p_mode="additive") if kind == "p" else \
        dict(p, u_mask=mask, uy=1e-6 * signal, u_mode="additive")


def test_source_spectra_stay_after_the_source():
    from kwave_gb300 import _lib
    from kwave_gb300.solver import Simulation, SimulationBatch

    members = [((20, 18, 24), "p", 5), ((15, 21, 25), "u", 9), ((16, 12, 14), "p", 50)]
    probs = [_problem(i, *m) for i, m in enumerate(members)]

    def spectrum(sim, kind):
        n0, n1, n2 = sim.S.shape
        out = np.empty(2 * n0 * n1 * ((n2 // 2 + 2) // 2 * 2), np.float32)
        slot = 0 if kind == "p" else 4  # KW_S_P0, KW_S_U1
        _lib.check(_lib.lib().kw_plan_read_source_spectrum(sim._plan.handle, slot, _lib.ptr(out), out.size))
        return out

    batch = SimulationBatch.from_problems(probs)
    try:
        got = batch.run()
        spectra = [spectrum(s, m[1]) for s, m in zip(batch.sims, members)]
    finally:
        batch.close()
    for p, m, g, s in zip(probs, members, got, spectra):
        sim = Simulation.from_problem(p)
        try:
            want = sim.run()
            assert np.array_equal(g["p"], want["p"]) and np.abs(want["p"]).max() > 0
            assert np.array_equal(s, spectrum(sim, m[1])), m
        finally:
            sim.close()
