"""GPU: the FP64 block product (FP64 matrix instructions on factors read in the
operand layout) against the single-vector kernels, column by column, at the
edges of its tiles: one slab, partial row groups, rank remainders, one column
more than a block, segments of odd length and start."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# both sum the same FP64 products in another order: at most n + k terms of
# relative size 1, so n eps = 1e-12 at worst and 1e-14 in practice
@pytest.mark.parametrize("n,dim,tree", [(40, 1, "bisect"), (1000, 1, "kmeans"), (5003, 1, "bisect"), (6001, 2, "bisect"),
                                        (8192, 1, "bisect")])
@pytest.mark.parametrize("ncols", [2, 7, 9, 16, 17, 33])
def test_block_vs_single(n, dim, tree, ncols):
    import hmatrix as hm
    rng = np.random.default_rng(n)
    geom = np.sort(rng.uniform(0, 10, n)) if dim == 1 else rng.uniform(0, 1, (n, 2))
    _, H = hm.NewHmat(hm.Params(Geom=geom, Kernel=hm.Cauchy(0.7), MaxBlock=min(512, n), MinBlock=64, MaxRank=16,
                                ConsMethod="aca2", εComp=1e-8, Tree=tree))
    X = rng.standard_normal((n, ncols))
    for trans in (False, True):
        Y = H.matvec(X, trans=trans)
        for j in range(ncols):
            y = H.matvec(np.ascontiguousarray(X[:, j]), trans=trans)
            assert np.linalg.norm(Y[:, j] - y) <= 1e-13 * np.linalg.norm(y)
