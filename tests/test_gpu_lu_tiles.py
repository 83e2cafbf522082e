"""GPU: the tile schedule's dense diagonal tiles against the recursion (lu! as
written) on the same H-matrix: the same pivots, the same L\\U up to the
truncation, the same solutions, for leaf sizes at the edges of the LU kernel's
panels (up to 32, 64 and more rows) and tiles that are not whole 32-row blocks,
every storage, and solves of one, several and more than 64 columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# both schedules truncate at eps_trunc = 1e-10 relative to a block: the packed
# factors agree to 1e-9 (as the oracle test asks), the solutions of the well
# conditioned system (shift 1, |H| < n) to 1e-8
@pytest.mark.parametrize("n,minb,maxb", [(1000, 16, 128), (1500, 32, 256), (2300, 64, 512), (1111, 70, 300), (900, 140, 300)])
def test_tiles_vs_recursion(n, minb, maxb):
    import hmatrix as hm
    rng = np.random.default_rng(n)
    prm = dict(Geom=np.sort(rng.uniform(0, 10, n)), Kernel=hm.Cauchy(1.0), MaxBlock=maxb, MinBlock=minb, MaxRank=16,
               ConsMethod="aca2", εComp=1e-10, Tree="bisect", Shift=1.0)
    _, H = hm.NewHmat(hm.Params(LuMode="tiles", **prm))
    _, G = hm.NewHmat(hm.Params(LuMode="recursive", **prm))
    L, R = hm.lu(H), hm.lu(G)
    assert L.info().lu_tiles >= 2 and R.info().lu_tiles == 0
    assert np.array_equal(L.P, R.P)
    A, B = L.to_dense(), R.to_dense()
    assert np.abs(A - B).max() <= 1e-9 * np.abs(B).max()
    for nc in (1, 5, 70):
        y = rng.standard_normal((n, nc))
        for trans in (False, True):
            x, z = L.solve(y, trans=trans), R.solve(y, trans=trans)
            assert np.linalg.norm(x - z) <= 1e-8 * np.linalg.norm(z)


@pytest.mark.parametrize("storage", ["F32"])
def test_tiles_from_reduced_storage(storage):
    """The stored (rounded) factors are what is factorised: refinement on the
    same handle reaches its FP64 target.  (BF16 factors are outside: their
    rounding is noise at full rank, and lu! at 1e-10 reports HM_ERR_RANK.)"""
    import hmatrix as hm
    n = 3000
    _, H = hm.NewHmat(hm.Params(Geom=np.linspace(0, 10, n), Kernel=hm.Cauchy(1.0), MaxBlock=256, MinBlock=32, MaxRank=12,
                                ConsMethod="aca2", εComp=1e-10, Tree="bisect", Shift=1.0, Storage=getattr(hm, storage)))
    y = np.random.default_rng(1).standard_normal(n)
    L = hm.lu(H)
    assert L.info().lu_tiles >= 2
    x, it, rr = L.solve_refined(y, tol=1e-12, max_iter=10)
    assert rr <= 1e-12


# a sweep step keeps the first 384 rows of a tile's dot products and the first
# 24 columns of each row segment in registers and loads the rest later: tiles
# on both sides, ragged ones, and the one-column path against the many-column
# one.  The same factors, so only rounding separates the two: the condition
# number (|H| < n, shift 1) times 2^-53 times a growth of 100.
@pytest.mark.parametrize("n,maxb", [(700, 128), (1537, 384), (1999, 512), (4100, 1024), (3000, 100)])
def test_sweep_columns(n, maxb):
    import hmatrix as hm
    rng = np.random.default_rng(n)
    _, H = hm.NewHmat(hm.Params(LuMode="tiles", Geom=np.sort(rng.uniform(0, 10, n)), Kernel=hm.Cauchy(1.0), MaxBlock=maxb,
                                MinBlock=32, MaxRank=16, ConsMethod="aca2", εComp=1e-10, Tree="bisect", Shift=1.0))
    L = hm.lu(H)
    assert L.info().lu_tiles >= 2
    tol = n * 2.0 ** -53 * 100
    Y = rng.standard_normal((n, 64))
    for trans in (False, True):
        one = np.stack([L.solve(Y[:, j], trans=trans) for j in range(64)], axis=1)
        for nc in (2, 8, 9, 64):
            X = L.solve(Y[:, :nc], trans=trans)
            assert np.linalg.norm(X - one[:, :nc]) <= tol * np.linalg.norm(X)
        assert np.array_equal(one[:, 0], L.solve(Y[:, 0], trans=trans))
