"""Batches with an SM for every strand take the narrowest CTA without probing.
At the edges of the CTA widths and of the recording cadence they give the bits
of the widest CTA, and the pseudo-ECG is the sum over the recorded V."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lq():
    import lqt1_gb300 as lq
    lq.lib()
    return lq


def run(lq, n, nstrand, rec_every, threads, precision, t_stop):
    specs = [lq.InstanceSpec(types=np.full(n + (i % 2 if n > 2 else 0), lq.MCELL, np.uint8), bcl=400.0, s1_start=0.0,
                             s1_duration=1.0, s1_strength=-80.0, n_stim=1, dx=0.15, t_stop=t_stop, record=i == 0,
                             ecg_x0=0.15 * n + 5.0) for i in range(nstrand)]
    b = lq.Batch(specs, [lq.model("default")], precision=precision, max_beats=2, rec_every=rec_every, threads=threads)
    b.run()
    assert b.num_bad() == 0
    r = b.record(0)
    return b.config(), [b.get_state(), b.detect()["t_act"], r["v"], r["t"], r["ecg"]]


@pytest.mark.parametrize("n,nstrand,rec_every,precision,width", [
    (2, 1, 1, "MIXED", 128), (33, 3, 3, "MIXED", 128), (127, 2, 10, "MIXED", 128), (128, 1, 7, "MIXED", 128),
    (129, 1, 10, "MIXED", 256), (255, 2, 1, "MIXED", 256), (257, 1, 4, "MIXED", 512), (128, 1, 7, "FP64", 128),
    (40, 800, 9, "MIXED", None)])
def test_narrow_cta_equals_wide(lq, n, nstrand, rec_every, precision, width):
    prec, t_stop = getattr(lq, precision), 4.0
    cfg, a = run(lq, n, nstrand, rec_every, 0, prec, t_stop)
    if width:
        assert cfg["threads"] == width and cfg["min_ctas_per_sm"] == 1
    _, w = run(lq, n, nstrand, rec_every, 512, prec, t_stop)
    for x, y in zip(a, w):
        assert np.array_equal(x, y)
    v, ecg = a[2], a[4]
    assert len(v) in (-(-200 // rec_every), -(-201 // rec_every))   # 4 ms / 0.02 ms, time summed in floating point
    dv = np.gradient(v, axis=1)                             # one-sided at the ends, centred inside
    term = -dv / (np.arange(n) * 0.15 - (0.15 * n + 5.0))**2
    # a term is a few roundings of 1.1e-16, their sum up to n more
    assert (np.abs(ecg - term.sum(axis=1)) <= (n + 8) * 1.2e-16 * np.abs(term).sum(axis=1)).all()
