"""GPU: the FP64 block product's table of factor columns by input segment, which
the device makes: leaves of more columns than a tile (32), segments that fill a
tile exactly or by one more, blocks of rank zero, a matrix without low-rank
leaves.  Against the single-vector kernels, and the same bits on every handle
(the order of a segment's leaves in the table is left open)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    "rank64": dict(n=1500, dim=2, ConsMethod="bbfmm", MaxRank=8, MaxBlock=300, MinBlock=100, kernel="cauchy", p=1.0),
    "rank32": dict(n=1200, dim=1, ConsMethod="bbfmm", MaxRank=32, MaxBlock=300, MinBlock=150, kernel="cauchy", p=1.0),
    "rank11": dict(n=1200, dim=1, ConsMethod="bbfmm", MaxRank=11, MaxBlock=200, MinBlock=40, kernel="cauchy", p=1.0),
    "zero": dict(n=2200, dim=1, ConsMethod="aca2", MaxRank=32, MaxBlock=256, MinBlock=32, kernel="gauss", p=0.02),
    "dense": dict(n=300, dim=1, ConsMethod="aca2", MaxRank=8, MaxBlock=300, MinBlock=300, kernel="cauchy", p=1.0),
}


# both sum the same FP64 products in another order: at most n + k terms of
# relative size 1, so n eps = 1e-12 at worst and 1e-14 in practice
@pytest.mark.parametrize("name", list(CASES))
def test_columns(name):
    import hmatrix as hm
    c = dict(CASES[name])
    n, dim, kernel, p = c.pop("n"), c.pop("dim"), c.pop("kernel"), c.pop("p")
    rng = np.random.default_rng(n)
    geom = np.sort(rng.uniform(0, 10, n)) if dim == 1 else rng.uniform(0, 1, (n, 2))
    prm = hm.Params(Geom=geom, Kernel={"cauchy": hm.Cauchy, "gauss": hm.Gauss}[kernel](p), εComp=1e-8, Tree="bisect", **c)
    H, G = hm.NewHmat(prm)[1], hm.NewHmat(prm)[1]
    X = rng.standard_normal((n, 17))
    for trans in (False, True):
        Y = H.matvec(X, trans=trans)
        assert np.array_equal(Y, G.matvec(X, trans=trans))
        for j in range(17):
            y = H.matvec(np.ascontiguousarray(X[:, j]), trans=trans)
            assert np.linalg.norm(Y[:, j] - y) <= 1e-13 * np.linalg.norm(y)
