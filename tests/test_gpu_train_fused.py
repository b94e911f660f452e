"""The fused training step at the edges of its tiling (one 16-row batch, a
partial tile, exactly one tile, one tile per SM and several tiles per CTA), and
the gather of its inputs from buffers of any 4-byte alignment.

Gradients against the FP64 reference (which rounds activations to BF16 as the
kernel does): the relative 1e-2 of the norm of test_gpu_mlp.py, a few BF16
roundings (2^-9) of the propagated gradients."""
import numpy as np
import pytest

from oracle import mlp_ref

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("batch", [16, 112, 128, 144, 152 * 128, 2 * 152 * 128 + 80])
def test_gradients(batch):
    from lqt1_gb300.surrogate import Mlp
    m = Mlp(seed=7)
    rng = np.random.default_rng(batch)
    x = rng.normal(0, 1, (batch, 48)).astype(np.float32)
    t = rng.normal(0, 1, (batch, 48)).astype(np.float32)
    xd = torch.from_numpy(x).cuda().bfloat16()
    td = torch.from_numpy(t).cuda()
    loss = m.gradients(xd, td)
    g = m.grads()
    lref, gref = mlp_ref.loss_and_grads(m.params().astype(np.float64), x, t)
    assert abs(loss - lref) / lref < 1e-3
    assert np.linalg.norm(g - gref) / np.linalg.norm(gref) < 1e-2
    # every weight matrix and bias by itself
    for a, b in ((0, 6144), (6144, 6272), (6272, 22656), (22656, 22784), (22784, 28928), (28928, 28976)):
        assert np.linalg.norm(g[a:b] - gref[a:b]) / np.linalg.norm(gref[a:b]) < 2e-2, (a, b)
    # the same bits again, and from targets that are only 4-byte aligned
    m.gradients(xd, td)
    np.testing.assert_array_equal(m.grads(), g)
    buf = torch.empty(batch * 48 + 1, device="cuda")
    buf[1:] = td.reshape(-1)
    loss2 = m.gradients(xd, buf[1:].view(batch, 48))
    np.testing.assert_array_equal(m.grads(), g)
    assert loss2 == loss


@pytest.mark.parametrize("n", [1, 15, 16, 17, 5003])
@pytest.mark.parametrize("gather", [False, True])
def test_prepare(n, gather):
    from lqt1_gb300 import _native as N
    from lqt1_gb300 import surrogate as S
    L = S._bind_sur()
    rng = np.random.default_rng(n)
    rows = n + 7
    X = torch.from_numpy(rng.normal(0, 2, (rows, 44)).astype(np.float32)).cuda()
    D = torch.from_numpy(rng.normal(0, 1, (rows, 38)).astype(np.float32)).cuda()
    mean, scale, out = (rng.normal(0, 1, 48).astype(np.float32), rng.uniform(0.5, 2, 48).astype(np.float32),
                        rng.uniform(0.5, 2, 48).astype(np.float32))
    m = S.Mlp(seed=1)
    m.set_norm(mean, scale, out)
    idx = torch.from_numpy(rng.integers(0, rows, n)).cuda() if gather else None
    pick = idx if gather else torch.arange(n, device="cuda")
    mu, sc, os_ = (torch.from_numpy(a).cuda() for a in (mean, scale, out))
    want_x = torch.zeros(n, 48, device="cuda")
    want_x[:, :44] = (X[pick] - mu[:44]) * sc[:44]
    want_t = torch.zeros(n, 48, device="cuda")
    want_t[:, :38] = D[pick] / os_[:38]

    def call(shift):
        hold = [torch.empty(a.numel() + 4, dtype=a.dtype, device="cuda") for a in (X, D)]
        xs, ds = (h[shift:shift + a.numel()].view(a.shape) for h, a in zip(hold, (X, D)))
        xs.copy_(X)
        ds.copy_(D)
        xb = torch.full((n * 48 + 8,), -3.0, dtype=torch.bfloat16, device="cuda")
        t = torch.full((n * 48 + 8,), -3.0, device="cuda")
        N.check(L.lqt_sur_prepare(m._h, xs.data_ptr(), ds.data_ptr(), None if idx is None else idx.data_ptr(), n,
                                  xb[shift:].data_ptr(), t[shift:].data_ptr()), "lqt_sur_prepare")
        torch.cuda.synchronize()
        assert bool((xb[shift + n * 48:] == -3.0).all()) and bool((t[shift + n * 48:] == -3.0).all())
        return xb[shift:shift + n * 48].view(n, 48), t[shift:shift + n * 48].view(n, 48)

    for shift in (0, 1):
        xb, t = call(shift)
        assert bool((xb == want_x.bfloat16()).all())
        assert bool((t == want_t).all())
    # inputs alone
    xb = torch.empty((n, 48), dtype=torch.bfloat16, device="cuda")
    N.check(L.lqt_sur_prepare(m._h, X.data_ptr(), None, None if idx is None else idx.data_ptr(), n, xb.data_ptr(), None),
            "lqt_sur_prepare")
    torch.cuda.synchronize()
    assert bool((xb == want_x.bfloat16()).all())
