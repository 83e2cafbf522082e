"""GPU: phase 2 of the single-column product by row slabs (the default below
n = 2^18 and off the 64-row grid) against the window shapes on the same
factors, at sizes where slabs and leaves end anywhere: one slab, a slab of one
row more than a warp, leaves read along their rows (H'x), every storage."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# FP64: the same products in another order (n eps at most; 1e-14 as for the
# other shapes).  FP32/BF16: FP32 partial sums of at most 16 terms in either
# shape, 16 * 2^-24 = 1e-6 of the sum of magnitudes (here within 4 of |y|).
TOL = {"F64": 1e-14, "F32": 4e-6, "BF16": 4e-6}


@pytest.mark.parametrize("storage", ["F64", "F32", "BF16"])
@pytest.mark.parametrize("n,dim", [(33, 1), (1000, 1), (5003, 1), (40011, 1), (7001, 2)])
def test_slabs_vs_windows(n, dim, storage):
    import hmatrix as hm
    rng = np.random.default_rng(n)
    geom = np.sort(rng.uniform(0, 10, n)) if dim == 1 else rng.uniform(0, 1, (n, 2))
    _, H = hm.NewHmat(hm.Params(Geom=geom, Kernel=hm.Cauchy(0.7), MaxBlock=min(512, n), MinBlock=64, MaxRank=16,
                                ConsMethod="aca2", εComp=1e-8, Tree="bisect", Storage=getattr(hm, storage)))
    assert H.info().tune_p2_split == 1
    x = rng.standard_normal(n)
    got = [H * x, H.matvec(x, trans=True)]
    H.set_tune(4)
    for g, w in zip(got, [H * x, H.matvec(x, trans=True)]):
        assert np.linalg.norm(g - w) <= TOL[storage] * np.linalg.norm(w)


def test_rows_without_a_leaf_stay_finite():
    """A slab entry covers some of the slab's rows: an infinite z value must
    not reach the others (a row shard's rows outside its range have no leaf)."""
    import hmatrix as hm
    n = 4096
    _, H = hm.NewHmat(hm.Params(Geom=np.linspace(0, 10, n), Kernel=hm.Cauchy(1.0), MaxBlock=512, MinBlock=64,
                                MaxRank=16, ConsMethod="aca2", εComp=1e-8, Tree="bisect", RowRange=(512, 1024)))
    x = np.ones(n)
    x[7] = np.inf
    y = H * x
    assert not y[:512].any() and not y[1024:].any() and not np.isfinite(y[512:1024]).any()
