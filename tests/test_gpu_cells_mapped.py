"""The cell interface on both sides of the size up to which its inputs and
outputs stay in page-locked host memory, and batch states and detectors in
input order: the same bits on both sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGE = 512


@pytest.fixture(scope="module")
def lq():
    import lqt1_gb300 as lq
    lq.lib()
    return lq


def drive(lq, n, precision):
    rng = np.random.default_rng(3)
    types = rng.integers(0, 5, EDGE + 1).astype(np.uint8)[:n]
    ist, gap = rng.uniform(-40, 0, EDGE + 1)[:n], rng.uniform(-2, 2, EDGE + 1)[:n]
    v0 = rng.uniform(-95, 20, EDGE + 1)[:n]
    c = lq.TPORdCells(types, precision=precision)
    out = [c.get_v(), c.get_dvdt(), c.get_currents()]
    assert np.array_equal(out[0], c.get_state()[:, 0]) and not out[1].any() and not out[2].any()
    for k in range(3):
        c.set_istim(ist if k < 2 else 0.0)
        c.set_dvgap_dt(gap)
        c.update(1 + k)
        out += [c.get_v(), c.get_dvdt(), c.get_currents(), c.get_state()]
        assert np.array_equal(out[-4], out[-1][:, 0])
    s = out[-1].copy()
    s[:, 0] = v0
    c.set_state(s)
    out += [c.get_v(), c.get_dvdt(), c.get_currents()]      # V of the new state, the rest of the last update
    assert np.array_equal(out[-3], v0 if precision == lq.FP64 else v0.astype(np.float32))
    c.update(2)
    return out + [c.get_v(), c.get_state()]


@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
def test_mapped_equals_device(lq, precision):
    prec = getattr(lq, precision)
    big = drive(lq, EDGE + 1, prec)
    for n in (1, 33, EDGE):
        for a, b in zip(drive(lq, n, prec), big):
            assert np.array_equal(np.asarray(a).reshape(n, -1), np.asarray(b).reshape(EDGE + 1, -1)[:n]), n


@pytest.mark.parametrize("precision", ["MIXED", "FP64"])
def test_batch_in_input_order(lq, precision):
    """Uneven instances (reordered inside) against each alone."""
    prec, n = getattr(lq, precision), [1, 130, 7, 1, 64, 300, 2]
    specs = [lq.InstanceSpec(types=np.full(k, (lq.ENDO, lq.EPI, lq.MCELL)[i % 3], np.uint8), bcl=300.0, s1_start=0.0,
                             s1_strength=-80.0, n_stim=3, t_stop=6.0 + i) for i, k in enumerate(n)]
    rng = np.random.default_rng(1)
    b = lq.Batch(specs, [lq.model("default")], precision=prec, max_beats=3)
    s = b.get_state()
    s[:, 0] += rng.uniform(0, 5, len(s))
    b.set_state(s)
    first = b.get_state()
    assert np.array_equal(first[:, 0], s[:, 0] if prec == lq.FP64 else s[:, 0].astype(np.float32))
    b.run()
    got, det = b.get_state(), b.detect()
    for i, x in enumerate(specs):
        sl = slice(b.offsets[i], b.offsets[i + 1])
        one = lq.Batch([x], [lq.model("default")], precision=prec, max_beats=3)
        one.set_state(s[sl])
        one.run()
        assert np.array_equal(one.get_state(), got[sl]), i
        d = one.detect()
        for key in ("t_act", "apd90", "dvdt_max", "ead", "beats"):
            assert np.array_equal(d[key], det[key][sl]), (i, key)
