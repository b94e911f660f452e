"""The FP64 step (tpord_f64.cuh: table exponentials, corrected reciprocals,
rearranged terms) against the CPU oracle over the voltages it is used at and far
outside them, where its exponentials saturate.

Tolerance: every elementary result is within a few 2^-53 and a state is a sum of
at most some forty of them; currents cancel to V's derivative by up to 1e3, so
1e-10 relative to the largest of the state, its change and the summed current
magnitudes times dt (1e3 times above what that gives, 1e4 below FP32)."""
import numpy as np
import pytest

import lqt1_gb300 as lq
from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [0.005, 0.02, 0.2])
@pytest.mark.parametrize("vrange", [(-120.0, 80.0), (-250.0, 290.0), (-40.0 - 1e-9, -40.0 + 1e-9), (-1e-3, 1e-3)])
@pytest.mark.parametrize("n", [1, 63, 2049])
def test_step_against_oracle(n, vrange, dt):
    rng = np.random.default_rng(n)
    s0 = orc.random_states(n, seed=n + 1)
    s0[:, 0] = rng.uniform(*vrange, n)
    types = rng.integers(0, 5, n).astype(np.uint8)
    ist = rng.uniform(-52, 0, n)
    for om, lm in ((orc.model("default"), lq.model("default")),
                   (orc.model("lqt1", gks_scale=0.5), lq.model("lqt1", gks_scale=0.5))):
        ref = orc.cells_update(s0.copy(), types, om, dt=dt, ist=ist, nsteps=1)
        c = lq.TPORdCells(types, precision=lq.FP64, model=lm, dt=dt)
        c.set_state(s0)
        c.set_istim(ist)
        c.update(1)
        got, cur = c.get_state(), c.get_currents()
        c.close()
        assert np.all(np.isfinite(got))
        size = np.maximum(np.abs(ref), np.abs(s0))
        size[:, 0] += dt * (np.abs(cur[:, :5]).sum(1) + np.abs(cur[:, 5]) + 100.0)
        # the reference's e^x - 1 and this form's lose the same digits near V = 0, not the same bits
        lost = 1.0 if vrange[1] > 1 or vrange[1] < -1 else 1e6
        assert np.all(np.abs(got - ref) <= 1e-10 * lost * np.maximum(size, 1e-6))
