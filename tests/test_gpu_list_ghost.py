"""Inside a macro step the listed voxels' plain step and the mirror voxels in one
launch, against the two launches that larger grids use: lqt_sim_profile steps
with the separate kernels, so the same run stepped both ways has the same bits."""
import numpy as np
import pytest

import lqt1_gb300 as lq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 5), (33, 31), (64, 16), (1, 1, 1), (7, 9, 11), (12, 16, 21)])
def test_one_launch_equals_two(shape):
    t = np.pad(np.full(shape, lq.EPI, np.uint8), 1, constant_values=lq.EMPTY)
    if t.size > 1000:
        t[tuple(slice(n // 3, n // 3 + 2) for n in t.shape)] = lq.EMPTY     # sources with several mirror voxels
    a = np.linspace(0.1, 1.4, t.size).reshape(t.shape)
    f = np.stack([np.cos(a), np.sin(a), 0 * a], -1).astype(np.float32)
    s1 = np.zeros(t.shape, np.uint8)
    s1[1:3] = t[1:3] != lq.EMPTY
    res = []
    for separate in (False, True):
        sim = lq.Sim(t, 0.2, fibre=f, model=lq.model("baseline", pca_scale=1.5))
        sim.set_protocol(bcl=30.0, s1_mask=s1, s1_start=0.3, s1_duration=1.0)
        sim.set_surrogate(lq.surrogate.load())
        sim.tune(2)                       # the separate kernels of a large grid
        sim.substep_variant(5)
        sim.step(10)
        for _ in range(20):
            if separate:
                sim.profile(30)
            else:
                sim.step(30)
        d = sim.detect()
        res.append([sim.get_state(), sim.get_v(), d["t_act"], np.array([sim.check(), sim.time]),
                    np.array(list(sim.surrogate_stats().values()))])
        sim.close()
    for x, y in zip(*res):
        np.testing.assert_array_equal(x, y)
