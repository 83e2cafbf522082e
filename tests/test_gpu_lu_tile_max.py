"""GPU: the H-LU's tiles hold at most 2048 rows where the partition allows it:
larger admissible blocks are taken in parts.  The factors are the recursion's up
to the truncation, and solve the system."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def params(hm, n, maxb, **kw):
    geom = np.sort(np.random.default_rng(n).uniform(0, 10, n))
    return hm.Params(Geom=geom, Kernel=hm.Cauchy(20.0), MaxBlock=maxb, MinBlock=128, MaxRank=6, ConsMethod="bbfmm",
                     Tree="bisect", Shift=1.0, εTruncLU=1e-10, **kw)


# MaxBlock of two halves, quarters; an odd size
@pytest.mark.parametrize("n,maxb,tiles", [(4096, 2048, 2), (4098, 2049, 4), (8192, 4096, 4), (8191, 4096, 4)])
def test_tiles_of_at_most_2048_rows(n, maxb, tiles):
    import hmatrix as hm
    _, H = hm.NewHmat(params(hm, n, maxb, LuMode="tiles"))
    y = np.random.default_rng(0).standard_normal(n)
    L = hm.lu(H)
    assert L.info().lu_tiles == tiles
    x = L.solve(y)
    # truncation at 1e-10 relative to a block, |H| < n
    assert np.linalg.norm(H * x - y) <= 1e-9 * n ** 0.5 * np.linalg.norm(x)
    x, it, rr = L.solve_refined(y, tol=1e-13, max_iter=5)
    assert rr <= 1e-13 and it <= 2


def test_parts_against_recursion():
    import hmatrix as hm
    n = 4500
    L, R = (hm.lu(hm.NewHmat(params(hm, n, 2250, LuMode=mode))[1]) for mode in ("tiles", "recursive"))
    assert L.info().lu_tiles == 4 and np.array_equal(L.P, R.P)
    A, B = L.to_dense(), R.to_dense()
    assert np.abs(A - B).max() <= 1e-9 * np.abs(B).max()
