"""GPU: aca2 by warps (blocks of at most 128 rows and columns) and by CTAs
(larger ones) against the dense kernel matrix: sizes on both sides of the line
and of a CTA's threads, up to the largest number of steps, and every storage."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# a block stops at |a_r||b_r| <= eps |a_1||b_1| (the usual estimate of the
# remainder, good to a small factor): 100 eps of the whole matrix, at least
# 1e-10; FP32 and BF16 factors add their rounding, 2^-24 and 2^-9 an entry
@pytest.mark.parametrize("storage,rnd", [("F64", 0.0), ("F32", 2.0 ** -24), ("BF16", 2.0 ** -9)])
@pytest.mark.parametrize("n,maxb,rank,tol,dim", [(1016, 127, 24, 1e-8, 1), (1032, 129, 24, 1e-8, 1), (2000, 250, 24, 1e-8, 1),
                                                 (1100, 550, 24, 1e-8, 1), (1600, 400, 64, 1e-30, 2)])
def test_blocks(storage, rnd, n, maxb, rank, tol, dim):
    import hmatrix as hm
    rng = np.random.default_rng(n)
    G = np.sort(rng.uniform(0, 10, n)) if dim == 1 else rng.uniform(0, 1, (n, 2))
    c, H = hm.NewHmat(hm.Params(Geom=G, Kernel=hm.Cauchy(1.0), MaxBlock=maxb, MinBlock=32, MaxRank=rank,
                                ConsMethod="aca2", εComp=tol, Tree="bisect", Shift=0.5, Storage=getattr(hm, storage)))
    A = hm.FullMat(hm.Cauchy(1.0), c.X, c.X) + 0.5 * np.eye(n)
    assert H.info().n_rk > 0
    assert np.linalg.norm(H.to_dense() - A) <= (max(100 * tol, 1e-10) + 4 * rnd) * np.linalg.norm(A)
