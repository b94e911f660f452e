"""Many steps of a small grid in one launch where its blocks are not ordered by
the V they exchange: two pieces of tissue without contact, grids of as many
blocks as the launch takes (and one voxel to either side), few steps per launch,
and several simulations side by side, so that blocks of a launch start far apart
in time.  Every voxel has to step with the clock of its own step (stimulus
windows, onsets, detector times): the same bits as one launch per step."""
import numpy as np
import pytest

import lqt1_gb300 as lq

pytestmark = pytest.mark.gpu


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def block(shape, extra=0):
    """shape voxels of tissue, `extra` more (or fewer) of them."""
    t = np.full(shape, lq.ENDO, np.uint8)
    t.reshape(-1)[::5] = lq.EPI
    if extra < 0:
        t.reshape(-1)[extra:] = lq.EMPTY
    if len(shape) == 1:
        return np.concatenate([t[t != lq.EMPTY], np.full(max(extra, 0), lq.ENDO, np.uint8)])
    if extra > 0:
        t = np.concatenate([t, np.full((1,) + t.shape[1:], lq.EMPTY, np.uint8)])
        t[-1].reshape(-1)[:extra] = lq.ENDO
    return np.pad(t, 1, constant_values=lq.EMPTY)


def islands(shape):
    t = block(shape)
    cut = t.shape[0] // 2
    t[cut:cut + 3] = lq.EMPTY
    return t


TISSUES = {
    "1d": lambda n: block((128 * n,)),
    "1d less": lambda n: block((128 * n - 1,)),
    "1d more": lambda n: block((128 * n + 1,)),
    "2d": lambda n: block((n, 128)),
    "2d less": lambda n: block((n, 128), -1),
    "2d more": lambda n: block((n, 128), 1),
    "3d": lambda n: block((n, 8, 16)),
    "3d more": lambda n: block((n, 8, 16), 1),
    "2d islands": lambda n: islands((n, 128)),
    "2d small islands": lambda n: islands((9, 40)),
    "3d islands": lambda n: islands((n, 8, 16)),
}


def make(t, stim):
    sim = lq.Sim(types=t, dx=0.18, model="default")
    s1 = t != lq.EMPTY
    on = np.random.default_rng(3).uniform(0, 0.2, t.shape).astype(np.float32) if stim == "onset" else None
    sim.set_protocol(bcl=0.7, s1_mask=s1, s1_start=0.06, s1_duration=0.1, s1_onset=on, s2_mask=s1, s2_time=0.5,
                     s2_duration=0.08, s2_strength=-30.0)
    return sim


def outputs(sim):
    sim.sync()
    d = sim.detect()
    out = [sim.get_state(), d["t_act"], d["apd90"], np.array([sim.check(), sim.time])]
    sim.close()
    return out


COUNTS = (4, 4, 6, 3, 10, 4, 5, 8, 4, 50)


@pytest.mark.parametrize("stim", ["window", "onset"])
@pytest.mark.parametrize("kind", sorted(TISSUES))
def test_every_block_steps_with_its_own_clock(kind, stim):
    t = TISSUES[kind](sms())
    ref = make(t, stim)
    ref.tune(2)
    ref.step(sum(COUNTS))
    want = outputs(ref)
    many = [make(t, stim) for _ in range(4)]
    for n in COUNTS:
        for sim in many:
            sim.step_async(n)
    for sim in many:
        for a, b in zip(outputs(sim), want):
            np.testing.assert_array_equal(a, b)


def broken():
    sim = make(islands((20, 30)), "window")
    sim.step(10)
    sim.set_wait_test(True, 2000)        # block 0 publishes nothing: its neighbours' waits run out
    return sim


def test_every_reader_reports_a_wait_that_ran_out(tmp_path):
    """Results of steps that did not complete are not handed out as if they had."""
    import torch
    sim = broken()
    sim.set_electrodes([(1.0, 1.0, 5.0)], every=50)
    host = torch.empty(sim.n, dtype=torch.float32).pin_memory()
    sim.step_async(10)
    sim.get_v_async(host.numpy())
    vtk = sim.vtk_writer(1)
    vtk.submit(str(tmp_path / "v.vtk"))
    for call in (lambda: sim.wait_v(upto=0), sim.wait_v, sim.sync, sim.get_v, sim.get_state, sim.detect, sim.ecg, sim.check,
                 lambda: sim.sample_v(1), lambda: sim.checkpoint(str(tmp_path / "c.bin")), vtk.flush,
                 lambda: sim.step_async(1), lambda: sim.step(2), lambda: sim.step(100),
                 lambda: sim.tune(-1), lambda: sim.profile(2)):
        with pytest.raises(lq.LqtError):
            call()
    vtk.close()
    assert not (tmp_path / "v.vtk").exists() and not (tmp_path / "c.bin").exists()
    sim.close()


def test_queued_launches_leave_once_a_wait_has_run_out():
    """With a bound of 2^21 polls per wait (0.3 s at the 150 ns of a poll), 40
    launches queued behind the one whose wait runs out would take over ten
    seconds; they end with it."""
    import time
    sim = broken()
    sim.set_wait_test(True, 1 << 21)
    t0 = time.perf_counter()
    with pytest.raises(lq.LqtError):
        for _ in range(40):
            sim.step_async(10)
        sim.sync()
    one = time.perf_counter() - t0
    sim.close()
    assert one < 5.0


def test_new_state_after_a_wait_that_ran_out(tmp_path):
    """A restored checkpoint runs on as it would have without the failure."""
    path = str(tmp_path / "c.bin")
    res = []
    for fail in (False, True):
        sim = make(islands((20, 30)), "window")
        sim.step(10)
        sim.checkpoint(path)
        if fail:
            sim.set_wait_test(True, 2000)
            sim.step_async(10)
            with pytest.raises(lq.LqtError):
                sim.sync()
            sim.set_wait_test(False)
            with pytest.raises(lq.LqtError):
                sim.step(4)
            sim.restore(path)
        sim.step(4)
        sim.step(20)
        res.append([sim.get_state(), np.array([sim.time])])
        sim.close()
    for a, b in zip(*res):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("every", [1, 2, 5, 10, 100])
def test_ecg_cadence(every):
    """Launches of many steps, replayed graphs and single steps take turns as the
    pseudo-ECG's cadence and the calls cut them: the same bits and samples."""
    t = islands((20, 30))
    res = []
    for forced in (False, True):
        sim = make(t, "window")
        sim.set_electrodes([(2.0, 3.0, 4.0)], every=every)
        if forced:
            sim.tune(2)
        for n in (3, 4, 43, 50, 100, 7, 93, 111):
            sim.step(n)
        res.append([sim.get_state(), *sim.ecg()])
        sim.close()
    for a, b in zip(*res):
        np.testing.assert_array_equal(a, b)
