"""GPU: the tensor-core block products' tiles (128 output rows, K blocks of Z
slots listed per tile) against the single-vector kernels column by column, at
sizes where a list goes wrong: clusters smaller than a tile and than a K block's
slots, a last tile of 1 and of 127 rows, fewer rows than a tile, one low-rank
leaf, every column-block width and both directions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# as for the other block products: FP32 accumulation of split products
TOL = {"F32": 1e-5, "BF16": 2e-5}


@pytest.mark.parametrize("storage", ["F32", "BF16"])
@pytest.mark.parametrize("n,minb,rank", [(96, 8, 3), (129, 8, 5), (1151, 16, 16), (4097, 12, 2), (3333, 100, 9), (257, 65, 1)])
def test_tile_lists(storage, n, minb, rank):
    import hmatrix as hm
    rng = np.random.default_rng(n)
    _, H = hm.NewHmat(hm.Params(Geom=np.sort(rng.uniform(0, 10, n)), Kernel=hm.Cauchy(1.0), MaxBlock=max(n // 2, minb),
                                MinBlock=minb, MaxRank=rank, ConsMethod="aca2", εComp=1e-9, Tree="bisect",
                                Storage=getattr(hm, storage)))
    for nc in (2, 16, 33, 64, 70):
        X = rng.standard_normal((n, nc))
        for trans in (False, True):
            Y = H.matvec(X, trans=trans)
            R = np.stack([H.matvec(X[:, j], trans=trans) for j in range(nc)], 1)
            assert np.linalg.norm(Y - R) <= TOL[storage] * np.linalg.norm(R), (nc, trans)
            assert np.abs(Y - R).max() <= 40 * TOL[storage] * np.abs(R).max(), (nc, trans)


# the dense leaves alone (one leaf is the whole matrix, or every leaf is full
# rank): FP64 sums of exact products of the stored FP32 entries
@pytest.mark.parametrize("n,minb", [(5, 8), (33, 64), (64, 64), (100, 128), (301, 301)])
def test_dense_leaves(n, minb):
    import hmatrix as hm
    rng = np.random.default_rng(n)
    _, H = hm.NewHmat(hm.Params(Geom=np.sort(rng.uniform(0, 10, n)), Kernel=hm.Cauchy(1.0), MaxBlock=minb, MinBlock=minb,
                                MaxRank=8, ConsMethod="aca2", εComp=1e-9, Tree="bisect", Storage=hm.F32))
    D = H.to_dense()
    for nc in (2, 7, 9, 16, 31, 64, 65):
        X = rng.standard_normal((n, nc))
        for A, trans in ((D, False), (D.T, True)):
            Y = H.matvec(X, trans=trans)
            assert np.abs(Y - A @ X).max() <= 8 * n * 2.0 ** -53 * (np.abs(A) @ np.abs(X)).max()
