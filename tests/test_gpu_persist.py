"""Many steps of a small grid in one launch (blocks of 128 voxels that exchange
V and wait for one another) against one launch per step: the same bits at the
edges of the blocks and of the launches, with S1, onsets, S2, detectors and the
pseudo-ECG; and a wait that runs out is reported."""
import numpy as np
import pytest

import lqt1_gb300 as lq

pytestmark = pytest.mark.gpu


def tissue(shape, fibre):
    t = np.array([lq.ENDO, lq.MCELL, lq.EPI], np.uint8)[np.arange(np.prod(shape)) % 3].reshape(shape)
    if len(shape) == 1:
        return dict(types=t, dx=0.15), np.arange(t.size) < 3
    if t.size > 200:
        t[tuple(slice(n // 3, n // 3 + max(1, n // 6)) for n in shape)] = lq.EMPTY
    t = np.pad(t, 1, constant_values=lq.EMPTY)
    kw = dict(types=t, dx=0.18)
    if fibre:
        a = np.linspace(0.1, 1.4, t.size).reshape(t.shape)
        kw["fibre"] = np.stack([np.cos(a), np.sin(a), 0 * a], -1).astype(np.float32)
    s1 = np.zeros(t.shape, bool)
    s1[1:3] = t[1:3] != lq.EMPTY
    return kw, s1


@pytest.mark.parametrize("shape,fibre", [((1,), False), ((2,), False), ((128,), False), ((129,), False), ((1000,), False),
                                         ((1, 1), False), ((8, 16), True), ((3, 43), False), ((53, 47), True),
                                         ((190, 200), False), ((1, 1, 1), True), ((4, 5, 13), True), ((13, 17, 29), True),
                                         ((24, 30, 50), False)])
@pytest.mark.parametrize("ecg", [0, 10])
def test_same_bits_as_single_steps(shape, fibre, ecg):
    kw, s1 = tissue(shape, fibre)
    res = []
    for forced in (False, True):
        sim = lq.Sim(model=lq.model("baseline", gks_scale=0.5, pca_scale=2.0), **kw)
        on = np.random.default_rng(1).uniform(0, 1, s1.shape).astype(np.float32) if ecg else None
        sim.set_protocol(bcl=9.0, s1_mask=s1, s1_start=0.4, s1_duration=1.0, s1_onset=on, s2_mask=np.flip(s1).copy(),
                         s2_time=5.0, s2_duration=0.5, s2_strength=-40.0)
        if ecg:
            sim.set_electrodes([(30.0, 3.0, 1.0)], every=ecg)
        if forced:
            sim.tune(2)
        for n in (2, 3, 7, 1, 500, 501, 89):
            sim.step_async(n)
        sim.sync()
        d = sim.detect()
        out = [sim.get_state(), sim.get_v(), d["t_act"], d["apd90"], np.array([sim.check(), sim.time])]
        res.append(out + (list(sim.ecg()) if ecg else []))
        sim.close()
    for a, b in zip(*res):
        np.testing.assert_array_equal(a, b)


def test_wait_that_runs_out_is_reported():
    kw, s1 = tissue((20, 30), True)
    sim = lq.Sim(**kw)
    sim.set_protocol(bcl=500.0, s1_mask=s1)
    sim.step(10)
    sim.set_wait_test(True, 2000)        # block 0 publishes nothing: its neighbours' waits run out
    with pytest.raises(lq.LqtError):
        sim.step(10)
    with pytest.raises(lq.LqtError):
        sim.step(10)
    sim.close()
    sim = lq.Sim(**kw)                   # the device works on
    sim.set_protocol(bcl=500.0, s1_mask=s1)
    sim.step(10)
    assert sim.check() == 0
    sim.close()
