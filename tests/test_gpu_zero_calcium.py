"""A calcium concentration of exactly zero (an empty sarcoplasmic store, subspace
or cytosol), or a store's far above any real one, in both forms of the cell step
against the FP64 oracle: the reference's formulas are finite there
(1 / (1 + K / 0) = 0, 1 / (1 + (1.5 / c)^8) = 1).

Tolerances: those of the same quantities in test_gpu_step_f32.py and
test_gpu_step_f64.py."""
import numpy as np
import pytest

import lqt1_gb300 as lq
from oracle import orc

pytestmark = pytest.mark.gpu

CAI, CASS, CAJSR = 5, 6, 8


@pytest.mark.parametrize("precision", [lq.MIXED, lq.FP64])
@pytest.mark.parametrize("zero", [0.0, -0.0])
@pytest.mark.parametrize("which", [(CAI,), (CASS,), (CAJSR,), (CAI, CASS, CAJSR)])
def test_zero_calcium(which, zero, precision):
    n = 257
    s0 = orc.random_states(n, seed=21)
    s0[:, 0] = np.linspace(-95.0, 45.0, n).astype(np.float32)
    s0[:, 9:] = s0[:, 9:].astype(np.float32)
    s0[:, list(which)] = zero
    types = np.arange(n).astype(np.uint8) % 5
    ref = orc.cells_update(s0.copy(), types, orc.model("default"), nsteps=1)
    assert np.all(np.isfinite(ref))
    c = lq.TPORdCells(types, precision=precision, model="default")
    c.set_state(s0)
    c.update(1)
    got, cur = c.get_state(), c.get_currents()
    c.update(50)
    later = c.get_state()
    c.close()
    assert np.all(np.isfinite(got)) and np.all(np.isfinite(later))
    total = np.abs(cur[:, :5]).sum(1) + np.abs(cur[:, 5])
    dt = 0.02
    if precision == lq.FP64:
        size = np.maximum(np.abs(ref), np.abs(s0))
        size[:, 0] += dt * (total + 100.0)
        assert np.all(np.abs(got - ref) <= 1e-10 * np.maximum(size, 1e-6))
        return
    gates = [j for j in range(9, 37) if j not in (12, 13)]
    assert np.abs(got[:, gates] - ref[:, gates]).max() <= 1e-5
    v = np.abs(s0[:, 0])
    dv = np.abs(got[:, 0] - ref[:, 0])
    assert np.all(dv <= 1e-5 * (np.abs(ref[:, 0] - s0[:, 0]) + dt * 4 * (total + v) + v) + 2e-5)
    for j in (37, 38):
        scale = np.maximum(np.abs(ref[:, j]), np.abs(s0[:, j]))
        assert np.all(np.abs(got[:, j] - ref[:, j]) <= 4e-5 * np.maximum(scale, 1e-9))


@pytest.mark.parametrize("precision", [lq.MIXED, lq.FP64])
@pytest.mark.parametrize("cajsr", [199.0, 201.0, 6e4, 7e4, 1e7, -1e7])
def test_large_store(cajsr, precision):
    s0 = orc.random_states(64, seed=22)
    s0[:, 9:] = s0[:, 9:].astype(np.float32)
    s0[:, CAJSR] = cajsr
    types = np.arange(64).astype(np.uint8) % 5
    ref = orc.cells_update(s0.copy(), types, orc.model("default"), nsteps=1)
    c = lq.TPORdCells(types, precision=precision, model="default")
    c.set_state(s0)
    c.update(1)
    got = c.get_state()
    c.close()
    assert np.all(np.isfinite(ref)) and np.all(np.isfinite(got))
    tol = 4e-5 if precision == lq.MIXED else 1e-12
    for j in (CAJSR, 37, 38):
        scale = np.maximum(np.abs(ref[:, j]), np.abs(s0[:, j]))
        assert np.all(np.abs(got[:, j] - ref[:, j]) <= tol * np.maximum(scale, 1e-9))


@pytest.mark.parametrize("precision", [lq.MIXED, lq.FP64])
def test_zero_calcium_on_tissue(precision):
    """The same through a simulation: no NaN, and as good as the cells alone."""
    sh = lq.geometry.sheet(20, 17)
    sim = lq.Sim(sh.types, 0.15, precision=precision)
    st = sim.get_state()
    st[:, [CAI, CASS, CAJSR]] = 0.0
    sim.set_state(st)
    sim.set_protocol(bcl=500.0, s1_mask=sh.s1_mask, s1_start=0.1)
    sim.step(100)
    assert sim.check() == 0 and np.all(np.isfinite(sim.get_state()))
    sim.close()
