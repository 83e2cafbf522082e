"""GPU: triangular solves with dense diagonal tiles by blocks of 32 rows (solves
of more than 64 columns, the panels of large tiles) at their edges: tiles of
whole and broken blocks, the largest that is solved in one piece (256 rows),
larger ones that are halved once or twice, a last block of one column.  The one-column solves
of the same factors multiply by the tiles' inverses instead."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the same factors, so only rounding separates the two: the condition number
# (|H| < n, shift 1) times 2^-53 times a growth of 100, as for the sweeps
@pytest.mark.parametrize("n,maxb", [(400, 100), (512, 128), (1203, 301), (1024, 256), (1028, 257), (2052, 513), (4400, 1100), (4393, 1100)])
def test_many_columns(n, maxb):
    import hmatrix as hm
    rng = np.random.default_rng(n)
    _, H = hm.NewHmat(hm.Params(LuMode="tiles", Geom=np.sort(rng.uniform(0, 10, n)), Kernel=hm.Cauchy(1.0), MaxBlock=maxb,
                                MinBlock=32, MaxRank=16, ConsMethod="aca2", εComp=1e-10, Tree="bisect", Shift=1.0))
    L = hm.lu(H)
    assert L.info().lu_tiles >= 4
    tol = n * 2.0 ** -53 * 100
    Y = rng.standard_normal((n, 97))
    for trans in (False, True):
        one = np.stack([L.solve(Y[:, j], trans=trans) for j in range(0, 97, 8)], axis=1)
        for nc in (65, 97):
            X = L.solve(Y[:, :nc], trans=trans)[:, ::8]
            assert np.linalg.norm(X - one[:, :X.shape[1]]) <= tol * np.linalg.norm(X)


# the panels against the recursion's (truncation at 1e-10, as for other tiles)
@pytest.mark.parametrize("n,maxb", [(1680, 840), (2600, 1300)])
def test_panels_of_large_tiles(n, maxb):
    import hmatrix as hm
    rng = np.random.default_rng(n)
    prm = dict(Geom=np.sort(rng.uniform(0, 10, n)), Kernel=hm.Cauchy(1.0), MaxBlock=maxb, MinBlock=64, MaxRank=16,
               ConsMethod="aca2", εComp=1e-10, Tree="bisect", Shift=1.0)
    L, R = (hm.lu(hm.NewHmat(hm.Params(LuMode=mode, **prm))[1]) for mode in ("tiles", "recursive"))
    assert L.info().lu_tiles >= 2 and np.array_equal(L.P, R.P)
    A, B = L.to_dense(), R.to_dense()
    assert np.abs(A - B).max() <= 1e-9 * np.abs(B).max()


# the recursion's leaves above the register kernels' 64 rows, against the dense
# solve (truncation at 1e-10, condition number below n)
@pytest.mark.parametrize("rows", [65, 75, 96, 97, 128, 159])
def test_leaves_of_the_recursion(rows):
    import hmatrix as hm
    n = 8 * rows
    rng = np.random.default_rng(rows)
    _, H = hm.NewHmat(hm.Params(LuMode="recursive", Geom=np.sort(rng.uniform(0, 10, n)), Kernel=hm.Cauchy(1.0),
                                MaxBlock=2 * rows, MinBlock=rows, MaxRank=16, ConsMethod="aca2", εComp=1e-10,
                                Tree="bisect", Shift=1.0))
    A = H.to_dense()
    L = hm.lu(H)
    for nc in (1, 33):
        Y = rng.standard_normal((n, nc))
        for M, trans in ((A, False), (A.T, True)):
            Z = np.linalg.solve(M, Y)
            assert np.linalg.norm(L.solve(Y, trans=trans) - Z) <= 1e-8 * np.linalg.norm(Z)
