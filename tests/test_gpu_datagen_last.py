"""A training pair drawn at a cell's very last macro step is written like every
other: with every boundary recorded (prob 1) and a cycle of whole macro steps,
the last row of each cell is such a pair, and a buffer filled with NaN keeps
none of it."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nsub", [1, 5, 10])
def test_last_pair_is_written(nsub):
    import ctypes as C

    from lqt1_gb300 import _native as N
    from lqt1_gb300 import surrogate as S
    L = S._bind_sur()
    ncells, cap = 7, 60_000
    X = torch.full((cap, 44), float("nan"), device="cuda")
    D = torch.full((cap, 38), float("nan"), device="cuda")
    two = C.c_double * 2
    r = S.SurRanges(two(0.5, 0.5), two(1.5, 1.5), two(1.2, 1.2), two(60.0, 60.0), 0, 1, 0.02, 1e9, 1.0, 0.0, nsub, 0)
    n = C.c_int64()
    N.check(L.lqt_sur_datagen(ncells, 3, C.byref(r), X.data_ptr(), D.data_ptr(), cap, C.byref(n), C.c_void_p(0)),
            "lqt_sur_datagen")
    assert 0 < n.value < cap and n.value % ncells == 0
    assert bool(torch.isfinite(X[:n.value]).all()) and bool(torch.isfinite(D[:n.value]).all())
    assert bool(torch.isnan(D[n.value:]).all())
