"""When the autotuner runs: a call of 64 steps starts it and steps 64 steps, with a
surrogate attached too; small grids, whose step is one launch of its own kernel,
have nothing to choose and say so."""
import numpy as np
import pytest

import lqt1_gb300 as lq

pytestmark = pytest.mark.gpu


def sheet(n, **kw):
    sh = lq.geometry.sheet(n, n)
    a = np.linspace(0.2, 1.3, sh.types.shape[1])[None, :] + 0 * sh.types
    f = np.stack([np.cos(a), np.sin(a), 0 * a], -1).astype(np.float32)
    sim = lq.Sim(types=sh.types, fibre=f, dx=0.15, model=lq.model("baseline", gks_scale=0.5, pca_scale=2.0, gks_iso_scale=1.5), **kw)
    sim.set_protocol(bcl=500.0, s1_mask=sh.s1_mask)
    return sim


@pytest.mark.parametrize("nsteps", [63, 64, 74, 75, 100])
def test_call_that_starts_it(nsteps):
    sim = sheet(300)                     # above the small grids (77,824 voxels at 152 SMs)
    sim.set_surrogate(lq.surrogate.load())
    sim.step(nsteps)
    assert abs(sim.time - 0.02 * nsteps) < 1e-9
    ms = sim.substep_variant(-1, timings=True)[1]
    assert bool((np.asarray(ms) > 0).all()) == (nsteps >= 64)
    sim.close()


@pytest.mark.parametrize("n", [40, 200])
def test_small_grid_has_nothing_to_choose(n):
    sim = sheet(n)
    sim.step(100)
    t0 = sim.time
    for _ in range(3):
        chosen, ms = sim.tune(-1)
        assert chosen == 2 and ms[0] > 0 and not ms[1:].any()
    assert sim.time > t0                 # real steps, as ever
    sim.close()
