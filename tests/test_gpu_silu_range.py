"""SiLU at pre-activations far outside the network's usual ones, in inference and
in training: x / (1 + exp(-x)) is 0 for any large negative x, x itself for a
large positive one, infinite for infinity and NaN for -infinity and NaN.

The network passes one activation through: X[r][0] = x, every other input 0,
first-layer weights +-1 in column 0, one unit read by the second layer, whose
bias of 50 keeps it in SiLU's linear part; output 50 + SiLU(x).  Tolerance: four
roundings to BF16 (2^-9 each) of values up to the larger of 50 and |x|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

HID, IN, OUT = 128, 48, 48
VALUES = [-3e38, -1e30, -1e20, -1e19, -1e4, -200.0, -104.0, -88.0, -82.0, -60.0, -44.0, -42.0, -41.0, -20.0, -1.0, 0.0, 1.0,
          44.0, 88.0, 1e4, 1e20, float("-inf"), float("inf"), float("nan")]


def bf16(a):
    return torch.tensor(a, dtype=torch.float32).bfloat16().float().numpy()


def silu(x):
    x = np.asarray(x, np.float64)
    with np.errstate(all="ignore"):
        return x / (1.0 + np.exp(-x))


def network(alternate, unit):
    """Parameters in the library's order W1 b1 W2 b2 W3 b3, weights [out][in]."""
    w1 = np.zeros((HID, IN), np.float32)
    w1[:, 0] = np.where(np.arange(HID) % 2 == 1, -1.0, 1.0) if alternate else 1.0
    w2 = np.zeros((HID, HID), np.float32)
    w2[:, unit] = 1.0
    w3 = np.zeros((OUT, HID), np.float32)
    w3[:, 3] = 1.0
    return np.concatenate([w1.ravel(), np.zeros(HID, np.float32), w2.ravel(), np.full(HID, 50.0, np.float32), w3.ravel(),
                           np.zeros(OUT, np.float32)])


@pytest.mark.parametrize("alternate", [False, True])
@pytest.mark.parametrize("unit", [0, 1, 31, 127])
@pytest.mark.parametrize("rows", [len(VALUES), 1000])
def test_inference(rows, unit, alternate):
    from lqt1_gb300.surrogate import Mlp
    m = Mlp(seed=1)
    m.set_params(network(alternate, unit))
    x = bf16([VALUES[r % len(VALUES)] for r in range(rows)])
    X = torch.zeros(rows, IN)
    X[:, 0] = torch.from_numpy(x)
    y = torch.empty(rows, OUT, device="cuda")
    m.infer(X.bfloat16().cuda(), y)
    got = y.cpu().numpy()
    pre = -x if alternate and unit % 2 == 1 else x
    finite = np.isfinite(x)
    want = silu(50.0 + silu(pre[finite]))
    size = np.maximum(50.0, np.abs(want))
    assert np.all(np.abs(got[finite] - want[:, None]) <= 4 * 2.0 ** -9 * size[:, None])
    assert not np.isfinite(got[~finite]).any()      # (weights of 0 times infinity)


def test_infinite_activation_stays_infinite():
    """No zero weight, every unit at +infinity: the output is infinite, not NaN."""
    from lqt1_gb300.surrogate import Mlp
    m = Mlp(seed=1)
    w1 = np.zeros((HID, IN), np.float32)
    w1[:, 0] = 1.0
    p = np.concatenate([w1.ravel(), np.zeros(HID, np.float32), np.full(HID * HID, 0.01, np.float32),
                        np.zeros(HID, np.float32), np.full(OUT * HID, -0.01, np.float32), np.zeros(OUT, np.float32)])
    m.set_params(p)
    X = torch.zeros(130, IN)
    X[:, 0] = float("inf")
    y = torch.empty(130, OUT, device="cuda")
    m.infer(X.bfloat16().cuda(), y)
    assert bool((y == float("-inf")).all())


def test_training():
    """The loss and the second layer's bias gradient with one activation at a
    large negative pre-activation, where SiLU and its derivative are 0."""
    from lqt1_gb300.surrogate import Mlp
    m = Mlp(seed=1)
    m.set_params(network(False, 0))
    for x in (-3e38, -3e32, -1e30, -1e20, -200.0, -88.0, -60.0):
        X = torch.zeros(128, IN)
        X[:, 0] = x
        t = torch.zeros(128, OUT)
        loss = m.gradients(X.bfloat16().cuda(), t.cuda())
        g = m.grads()
        # y = 50 in every valid column (nvalid = 38 of the 48): loss is their mean square
        assert abs(loss / 2500.0 - 1.0) <= 4 * 2.0 ** -9 * 2, x
        b1 = g[HID * IN: HID * IN + HID]
        assert np.all(np.abs(b1) <= 1e-18), x       # SiLU'(-60) = -5e-25, over 128 rows
        b2 = g[HID * IN + HID + HID * HID: HID * IN + HID + HID * HID + HID]
        assert np.all(np.isfinite(g)) and b2[3] > 0 and np.all(b2[np.arange(HID) != 3] == 0.0)
