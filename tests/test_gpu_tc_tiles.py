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
