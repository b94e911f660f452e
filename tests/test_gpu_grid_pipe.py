"""The pipelined step kernel (variant 100) gives the bits of the one-thread-per-
voxel kernels, at sizes around its tiles: fewer voxels than a warp, a partial
last tile, exactly one tile per resident warp (152 SMs x 16 warps x 32) and a
tile more, with and without fibres, with S1, S2 and detectors."""
import numpy as np
import pytest

import lqt1_gb300 as lq

pytestmark = pytest.mark.gpu


def run(variant, kw, s1, s2):
    sim = lq.Sim(model=lq.model("lqt1", gks_scale=0.5), **kw)
    sim.set_protocol(bcl=9.0, s1_mask=s1, s1_start=0.2, s1_duration=1.0, s1_strength=-52.0, s2_mask=s2, s2_time=3.0,
                     s2_duration=0.6, s2_strength=-40.0)
    sim.tune(variant)
    sim.step(7)
    sim.step(200)
    d = sim.detect()
    out = [sim.get_state(), d["t_act"], d["apd90"], np.array([sim.check()])]
    sim.close()
    return out


@pytest.mark.parametrize("nx,ny", [(5, 3), (31, 1), (33, 7), (257, 32), (608, 128), (609, 128)])
@pytest.mark.parametrize("fibre", [False, True])
def test_sheet(nx, ny, fibre):
    if ny < 2:
        ny = 2
    sh = lq.geometry.sheet(nx, ny)
    kw = dict(types=sh.types, dx=0.15)
    if fibre:
        a = np.linspace(0.1, 1.4, ny + 2)[None, :] + 0 * sh.types
        kw["fibre"] = np.stack([np.cos(a), np.sin(a), 0 * a], -1).astype(np.float32)
    want = run(2, kw, sh.s1_mask, sh.s2_mask)
    for a, b in zip(want, run(100, kw, sh.s1_mask, sh.s2_mask)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("nx,nz", [(40, 52), (90, 120)])
def test_shell(nx, nz):
    v = lq.geometry.ventricle(nx=nx, ny=nx, nz=nz, a_out=0.08 * nx, c_out=0.15 * nz, wall=0.03 * nx, z_base=0.17 * nz,
                              island_radius=0.02 * nx, stim_radius=0.03 * nx)
    kw = dict(types=v.types, fibre=v.fibre, dx=0.2)
    want = run(2, kw, v.s1_mask, v.s1_mask)
    for a, b in zip(want, run(100, kw, v.s1_mask, v.s1_mask)):
        np.testing.assert_array_equal(a, b)
