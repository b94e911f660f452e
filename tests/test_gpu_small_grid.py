"""The one-launch step of small grids (mirror voxels and clock in the step
kernel; inside a macro step the substep and the plain step of the listed voxels
in one kernel) against the separate kernels that a forced variant selects: the
same arithmetic, so the same bits, in 1D, 2D (with and without fibres) and 3D,
over S1, per-voxel onsets, S2, detectors and the pseudo-ECG."""
import numpy as np
import pytest

import lqt1_gb300 as lq

pytestmark = pytest.mark.gpu


def tissue(kind):
    if kind == "1d":
        t = np.array([lq.ENDO] * 40 + [lq.MCELL] * 31 + [lq.EPI] * 34, np.uint8)
        s1, s2 = np.zeros_like(t), np.zeros_like(t)
        s1[:3], s2[-4:] = 1, 1
        return dict(types=t, dx=0.15), s1, s2, [(60.0, 0.0, 0.0)]
    if kind.startswith("2d"):
        sh = lq.geometry.sheet(37, 29)
        # a hole and a notch: sources with several mirror voxels
        sh.types[10:13, 9:14] = lq.EMPTY
        sh.types[20, 1:5] = lq.EMPTY
        kw = dict(types=sh.types, dx=0.15)
        if kind == "2d-fibre":
            a = np.linspace(0.2, 1.3, sh.types.shape[1])[None, :] + 0 * sh.types
            kw["fibre"] = np.stack([np.cos(a), np.sin(a), 0 * a], -1).astype(np.float32)
        return kw, sh.s1_mask, sh.s2_mask, [(8.0, 8.0, 4.0)]
    v = lq.geometry.ventricle(nx=40, ny=40, nz=52, a_out=3.4, c_out=8.4, wall=1.4, z_base=9.4, island_radius=1.0,
                              stim_radius=1.2)
    return dict(types=v.types, fibre=v.fibre, dx=0.2), v.s1_mask, np.roll(v.s1_mask, 3, 0), [(12.0, 4.0, 5.0)]


@pytest.mark.parametrize("kind", ["1d", "2d", "2d-fibre", "3d"])
@pytest.mark.parametrize("sur", [False, True])
@pytest.mark.parametrize("onset", [False, True])
def test_same_bits_as_separate_kernels(kind, sur, onset):
    kw, s1, s2, el = tissue(kind)
    rng = np.random.default_rng(2)
    res = []
    for forced in (False, True):
        sim = lq.Sim(model=lq.model("baseline", gks_scale=0.5, pca_scale=2.0, gks_iso_scale=1.5), **kw)
        assert sim.n < 152 * 512
        on = rng.uniform(0, 2, s1.shape).astype(np.float32) if onset else None
        rng = np.random.default_rng(2)
        if onset:
            on = rng.uniform(0, 2, s1.shape).astype(np.float32)
        sim.set_protocol(bcl=12.0, s1_mask=s1, s1_start=0.5, s1_duration=1.0, s1_strength=-52.0, s1_beats=0,
                         s1_onset=on, s2_mask=s2, s2_time=6.0, s2_duration=1.0, s2_strength=-40.0)
        sim.set_electrodes(el, every=50)
        if sur:
            sim.set_surrogate(lq.surrogate.load())
        if forced:
            sim.tune(2)
            sim.substep_variant(5)
        sim.step(37)
        sim.step(250)
        for _ in range(23):
            sim.step_async(1)
        sim.sync()
        d = sim.detect()
        phi, t = sim.ecg()
        res.append([sim.get_state(), sim.get_v(), d["t_act"], d["apd90"], phi, t, np.array([sim.check()])] +
                   ([np.array(list(sim.surrogate_stats().values()))] if sur else []))
        sim.close()
    for a, b in zip(*res):
        np.testing.assert_array_equal(a, b)
