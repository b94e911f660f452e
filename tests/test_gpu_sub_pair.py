"""The substep kernels that take two voxels per thread (a producer warp's rows;
every warp its own rows), at the edges of their tiles of 256 and units of 64:
the bits of the one-voxel kernel, with plain voxels, stimuli and detectors
among them."""
import numpy as np
import pytest

import lqt1_gb300 as lq

pytestmark = pytest.mark.gpu


def tissue(shape):
    t = np.pad(np.full(shape, lq.MCELL, np.uint8), 1, constant_values=lq.EMPTY)
    a = np.linspace(0.1, 1.4, t.size).reshape(t.shape)
    c = 0.3 if t.ndim == 3 else 0.0
    f = np.stack([np.cos(a) * np.sqrt(1 - c * c), np.sin(a) * np.sqrt(1 - c * c), 0 * a + c], -1).astype(np.float32)
    s1 = np.zeros(t.shape, np.uint8)
    s1[1, ...] = t[1, ...] != lq.EMPTY
    return t, f, s1


@pytest.mark.parametrize("shape", [(1, 1), (1, 32), (3, 11), (9, 7), (8, 8), (5, 13), (15, 17), (16, 16), (1, 257), (31, 33),
                                   (1, 1, 1), (3, 3, 7), (4, 4, 4), (5, 13, 1), (4, 8, 8), (3, 11, 31), (8, 16, 24)])
def test_pair_kernels_same_bits(shape):
    types, fibre, s1 = tissue(shape)
    res = []
    for variant in (5, 304, 305, 306):
        sim = lq.Sim(types, 0.2, fibre=fibre, model=lq.model("baseline", pca_scale=1.5))
        s = sim.get_state()
        s[:, 0] += np.random.default_rng(4).uniform(0, 12, sim.n)
        sim.set_state(s)
        # the window opens inside a macro step; the second one finds most voxels on the plateau
        sim.set_protocol(bcl=6.0, s1_mask=s1, s1_start=0.5, s1_duration=0.7, s1_strength=-52.0, s1_beats=0)
        sim.set_surrogate(lq.surrogate.load())
        sim.tune(2)
        sim.substep_variant(variant)
        sim.step(430)
        d = sim.detect()
        res.append([sim.get_state(), sim.get_v(), d["t_act"], d["apd90"], np.array([sim.check()]),
                    np.array(list(sim.surrogate_stats().values()))])
        sim.close()
    for r in res[1:]:
        for a, b in zip(res[0], r):
            np.testing.assert_array_equal(a, b)
