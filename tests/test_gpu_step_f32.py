"""The mixed form's fast step (tpord_f32.cuh) against the FP64 oracle at the
voltages where its rewritten terms change form: the GHK polynomial's limit
(|V F/RT| = 0.5) and its value at V = 0, the INa branch at -40 mV, and far
outside the action potential, where the bounded exponentials saturate.

Tolerances: a gate is a convex combination of its old value and its steady
state, each within a few FP32 roundings of exponentials whose arguments stay
below 2^6 (argument rounding 2^-19, so 2e-6 of the value): 1e-5.  V: the
currents carry the same relative error; 1e-5 of the change in the step and of
the sum of the current magnitudes they are taken from, plus the rounding of V."""
import numpy as np
import pytest

import lqt1_gb300 as lq
from oracle import orc

pytestmark = pytest.mark.gpu

RT_F = 8314.0 * 310.0 / 96485.0
EDGES = np.array([0.0, 1e-6, -1e-6, 1e-3, -1e-3, 0.5 * RT_F, np.nextafter(np.float32(0.5 * RT_F), 100),
                  -0.5 * RT_F, 0.0026, -0.0026, -40.0, np.nextafter(np.float32(-40), 0), -40.00001])


@pytest.mark.parametrize("dt", [0.02, 0.2])
@pytest.mark.parametrize("vrange", [(-120.0, 80.0), (-250.0, 290.0)])
@pytest.mark.parametrize("n", [1, 33, 4099])
def test_step_against_oracle(n, vrange, dt):
    rng = np.random.default_rng(n)
    s0 = orc.random_states(n, seed=n)
    v = rng.uniform(*vrange, n)
    m = min(n, len(EDGES))
    v[:m] = EDGES[:m]
    s0[:, 0] = v.astype(np.float32)
    s0[:, 9:] = s0[:, 9:].astype(np.float32)
    types = rng.integers(0, 5, n).astype(np.uint8)
    for om, lm in ((orc.model("default"), lq.model("default")),
                   (orc.model("baseline", gks_scale=0.5, pca_scale=2.0, gks_iso_scale=1.5),
                    lq.model("baseline", gks_scale=0.5, pca_scale=2.0, gks_iso_scale=1.5))):
        # at V = 0 the reference's GHK terms are 0/0: its limit, 1e-6 mV away
        so = s0.copy()
        so[so[:, 0] == 0.0, 0] = 1e-6
        ref = orc.cells_update(so, types, om, dt=dt, nsteps=1)
        c = lq.TPORdCells(types, precision=lq.MIXED, model=lm, dt=dt)
        c.set_state(s0)
        c.update(1)
        got = c.get_state()
        cur = c.get_currents()
        c.close()
        assert np.all(np.isfinite(got))
        gates = [j for j in range(9, 37) if j not in (12, 13)]
        assert np.abs(got[:, gates] - ref[:, gates]).max() <= 1e-5
        total = np.abs(cur[:, :5]).sum(1) + np.abs(cur[:, 5]) + np.abs(v)
        dv = np.abs(got[:, 0] - ref[:, 0])
        assert np.all(dv <= 1e-5 * (np.abs(ref[:, 0] - s0[:, 0]) + dt * 4 * total + np.abs(v)) + 2e-5)


@pytest.mark.parametrize("precision", [lq.MIXED, lq.FP64])
@pytest.mark.parametrize("cajsr", [-0.05, -0.0124, -0.0122, -0.005, -1e-4, 1e-4, 0.005, 1.2])
def test_release_time_constant_at_any_jsr_calcium(cajsr, precision):
    """tau_rel = 4.75 / (1 + 0.0123 / cajsr) below 0.005 is 0.005, also where it
    is negative (TPORd.cc:962-969); the release gates against the oracle, to a
    few roundings of a relaxation that is complete within the step (1e-5 of the
    steady state in FP32, 1e-12 in FP64)."""
    s0 = orc.random_states(64, seed=9)
    s0[:, 8] = np.float32(cajsr)
    types = np.arange(64).astype(np.uint8) % 5
    ref = orc.cells_update(s0.copy(), types, orc.model("default"), nsteps=1)
    c = lq.TPORdCells(types, precision=precision, model="default")
    c.set_state(s0)
    c.update(1)
    got = c.get_state()
    c.close()
    tol = 1e-5 if precision == lq.MIXED else 1e-12
    for j in (37, 38):
        scale = np.maximum(np.abs(ref[:, j]), np.abs(s0[:, j]))
        assert np.all(np.abs(got[:, j] - ref[:, j]) <= tol * np.maximum(scale, 1e-9) * (1 if precision == lq.FP64 else 4))
