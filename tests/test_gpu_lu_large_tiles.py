"""GPU: the tile schedule's trailing updates on tiles of more rows than the
register kernels hold (512), at rank capacities so small that every pair would
fit their columns: each pair has to reach a kernel that takes it, or lu! returns
the factors of another matrix.  Against the recursion (lu! as written) on the
same H-matrix, with FP64 and with FP32 recompression cores."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# rank of the whole kernel matrix at 1e-10: 5 at l = 40, 4 at l = 160, so no
# capacity overflows.  Both schedules truncate at eps relative to a block: the
# packed factors agree to 10 eps, as for the other tile sizes; the pivots are
# the same (diagonal leaves are dominated by the shift), and the solutions of
# the well conditioned system (shift 1, |H| < n) to 100 eps.
@pytest.mark.parametrize("eps", [1e-10, 1e-6])
@pytest.mark.parametrize("n,maxb", [(2400, 600), (4400, 1100), (4393, 1100)])
@pytest.mark.parametrize("cap,ell", [(6, 40.0), (4, 160.0)])
def test_small_capacity(n, maxb, cap, ell, eps):
    import hmatrix as hm
    rng = np.random.default_rng(n + cap)
    prm = dict(Geom=np.sort(rng.uniform(0, 10, n)), Kernel=hm.Cauchy(ell), MaxBlock=maxb, MinBlock=64, MaxRank=cap,
               RankCap=cap, ConsMethod="aca2", εComp=1e-11, Tree="bisect", Shift=1.0, εTruncLU=eps)
    _, H = hm.NewHmat(hm.Params(LuMode="tiles", **prm))
    _, G = hm.NewHmat(hm.Params(LuMode="recursive", **prm))
    L, R = hm.lu(H), hm.lu(G)
    assert L.info().lu_tiles >= 4 and L.info().lu_rank_cap == cap
    assert np.array_equal(L.P, R.P)
    A, B = L.to_dense(), R.to_dense()
    assert np.abs(A - B).max() <= 10 * eps * np.abs(B).max()
    y = rng.standard_normal(n)
    for trans in (False, True):
        x, z = L.solve(y, trans=trans), R.solve(y, trans=trans)
        assert np.linalg.norm(x - z) <= 100 * eps * np.linalg.norm(z)
