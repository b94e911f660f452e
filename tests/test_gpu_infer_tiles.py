"""Tensor-core inference at the edges of its tiling: fewer rows than a tile, a
partial last tile, one tile per SM and more tiles than all groups of a launch
hold; an output buffer that is only 4-byte aligned; a row with a NaN input.

Tolerance: BF16 weights and two BF16 roundings of the activations (2^-9 each),
accumulated over 128 products: 2e-2 of the largest output, as for the
partial-tile check in test_gpu_mlp.py."""
import numpy as np
import pytest

from oracle import mlp_ref

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 152 * 128, 152 * 4 * 128 + 33, 3 * 152 * 4 * 128 - 1])
def test_rows(n):
    from lqt1_gb300.surrogate import Mlp
    m = Mlp(seed=5)
    rng = np.random.default_rng(n)
    x = torch.from_numpy(rng.normal(0, 1, (n, 48)).astype(np.float32)).cuda().bfloat16()
    guard = 64
    buf = torch.full((n * 48 + guard + 1,), -7.0, device="cuda")
    y = buf[: n * 48].view(n, 48)
    m.infer(x, y)
    pick = np.unique(np.concatenate([np.arange(min(n, 256)), np.arange(max(0, n - 256), n), rng.integers(0, n, 256)]))
    ref = mlp_ref.forward(m.params(), x[pick].float().cpu().numpy())["y"]
    got = y.cpu().numpy()
    assert np.abs(got[pick] - ref).max() < 2e-2 * np.abs(ref).max()
    assert bool((buf[n * 48:] == -7.0).all())
    # 4-byte aligned output, same bits
    odd = torch.full((n * 48 + guard + 1,), -7.0, device="cuda")
    m.infer(x, odd[1:1 + n * 48].view(n, 48))
    np.testing.assert_array_equal(odd[1:1 + n * 48].view(n, 48).cpu().numpy(), got)
    assert float(odd[0]) == -7.0 and bool((odd[1 + n * 48:] == -7.0).all())
    # a NaN stays in its row
    x2 = x.clone()
    x2[n // 2, 3] = float("nan")
    m.infer(x2, y)
    g2 = y.cpu().numpy()
    assert np.isnan(g2[n // 2]).all()
    keep = np.arange(n) != n // 2
    np.testing.assert_array_equal(g2[keep], got[keep])
