"""GPU: the largest diagonal leaves lu! takes.  Both schedules keep a leaf of up
to 159 rows in shared memory; beyond that they refuse it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def params(hm, n, minb, mode):
    rng = np.random.default_rng(n)
    return hm.Params(LuMode=mode, Geom=np.sort(rng.uniform(0, 10, n)), Kernel=hm.Cauchy(1.0), MaxBlock=2 * minb,
                     MinBlock=minb, MaxRank=16, ConsMethod="aca2", εComp=1e-10, Tree="bisect", Shift=1.0)


# the tolerances of the other tile sizes (truncation at 1e-10)
@pytest.mark.parametrize("rows", [151, 152, 159])
def test_leaves_up_to_159_rows(rows):
    import hmatrix as hm
    n = 8 * rows
    L, R = (hm.lu(hm.NewHmat(params(hm, n, rows, mode))[1]) for mode in ("tiles", "recursive"))
    assert L.info().lu_tiles >= 2 and R.info().lu_tiles == 0
    assert np.array_equal(L.P, R.P)
    A, B = L.to_dense(), R.to_dense()
    assert np.abs(A - B).max() <= 1e-9 * np.abs(B).max()


@pytest.mark.parametrize("mode", ["auto", "tiles", "recursive"])
def test_larger_leaves_are_refused(mode):
    import hmatrix as hm
    _, H = hm.NewHmat(params(hm, 8 * 160, 160, mode))
    with pytest.raises(hm.HmError) as ei:
        hm.lu(H)
    assert "above 159 rows" in str(ei.value)
