"""The macro step's tiles (state rows copied ahead in whole tiles of 128, the
last one ragged): without diffusion every voxel is on its own, so a voxel gives
the same bits wherever it stands -- first or last of a tile, in any tile of a
warpgroup's turn, alone in the last tile."""
import numpy as np
import pytest

import lqt1_gb300 as lq

pytestmark = pytest.mark.gpu


def library():
    """States of the three types over one paced beat."""
    types = np.array([lq.ENDO, lq.MCELL, lq.EPI], np.uint8)
    c, out = lq.TPORdCells(types), []
    for k in range(60):
        c.set_istim(-53.0 if k < 2 else 0.0)
        c.update(25 if k < 20 else 400)
        out.append(c.get_state())
    return types, np.stack(out)


@pytest.mark.parametrize("use_net", [True, False])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 640, 152 * 512 + 1, 2 * 152 * 512 - 127])
def test_place_in_the_grid_does_not_matter(n, use_net):
    types, lib = library()
    rng = np.random.default_rng(n)
    which, phase = rng.integers(0, 3, n), rng.integers(0, len(lib), n)
    state = lib[phase, which]
    state[:, 0] += rng.uniform(-0.5, 0.5, n)
    res = []
    inner = np.full(-(-n // 64) * 64, lq.EMPTY, np.uint8)        # rows of 64, the last one ragged
    inner[:n] = lq.ENDO
    sheet = np.pad(inner.reshape(-1, 64), 1, constant_values=lq.EMPTY)
    grid = sheet.reshape(-1)
    sim = lq.Sim(sheet, 0.15)
    index = sim.tissue_index()
    sim.close()
    for perm in (np.arange(n), rng.permutation(n)):
        grid[index] = types[which[perm]]
        sim = lq.Sim(sheet, 0.15, d_fibre=0.0, d_trans=0.0, model=lq.model("baseline", pca_scale=1.3))
        assert np.array_equal(sim.tissue_index(), index)
        sim.set_protocol(bcl=500.0, s1_mask=np.zeros(grid.shape, np.uint8), s1_start=400.0)
        sim.set_state(state[perm])
        sim.set_surrogate(lq.surrogate.load(), use_net=use_net)
        sim.step(20)
        assert sim.check() == 0
        s = np.empty_like(state)
        s[perm] = sim.get_state()
        d = sim.detect()
        t = np.empty_like(d["t_act"])
        t[perm] = d["t_act"]
        res.append((s, t, np.array(list(sim.surrogate_stats().values())), np.array(list(sim.surrogate_rejections().values()))))
        sim.close()
    for a, b in zip(*res):
        np.testing.assert_array_equal(a, b)
    assert n < 600 or 0 < res[0][2][2] <= res[0][2][1]
