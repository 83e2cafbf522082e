"""GPU: the row slab lists, which the device makes from the window lists, where a
window's end cuts a slab or a leaf: slabs astride a 1024-row boundary, leaves over
several windows and smaller than a slab, blocks of rank zero, leaves read along
their rows (H'x), a row shard whose other rows have no leaf.  Against the window
shape on the same factors, row by row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the same products in another order: n eps of the sum of their magnitudes,
# which |H| |x| bounds; an entry missed or taken twice is far outside
def check(hm, H, x, trans):
    y = H.matvec(x, trans=trans)
    assert H.info().tune_p2_split == 1
    D = H.to_dense()
    D = D.T if trans else D
    assert (np.abs(y - D @ x) <= 1e-12 * (np.abs(D) @ np.abs(x)) + 1e-300).all()


@pytest.mark.parametrize("n,minb,maxb,tree", [(1023, 64, 512, "bisect"), (1025, 8, 100, "bisect"), (3100, 30, 2048, "bisect"),
                                              (3100, 90, 700, "kmeans"), (2500, 300, 300, "bisect"), (4099, 1, 64, "bisect")])
def test_every_row(n, minb, maxb, tree):
    import hmatrix as hm
    rng = np.random.default_rng(n + minb)
    _, H = hm.NewHmat(hm.Params(Geom=np.sort(rng.uniform(0, 10, n)), Kernel=hm.Cauchy(0.5), MaxBlock=maxb, MinBlock=minb,
                                MaxRank=12, ConsMethod="aca2", εComp=1e-8, Tree=tree))
    x = rng.standard_normal(n)
    for trans in (False, True):
        check(hm, H, x, trans)


def test_blocks_of_rank_zero():
    """exp(-|x-y|^2 / (2 l^2)) underflows to zero away from the diagonal."""
    import hmatrix as hm
    n = 2200
    _, H = hm.NewHmat(hm.Params(Geom=np.linspace(0, 10, n), Kernel=hm.Gauss(0.02), MaxBlock=256, MinBlock=32, MaxRank=32,
                                ConsMethod="aca2", εComp=1e-8, Tree="bisect"))
    assert (H.leaves()[:, 0] == 1).any() and (H.leaves()[H.leaves()[:, 0] == 1][:, 5] == 0).any()
    x = np.random.default_rng(0).standard_normal(n)
    for trans in (False, True):
        check(hm, H, x, trans)


def test_row_shard():
    import hmatrix as hm
    n = 4096
    prm = dict(Geom=np.linspace(0, 10, n), Kernel=hm.Cauchy(1.0), MaxBlock=512, MinBlock=64, MaxRank=16, ConsMethod="aca2",
               εComp=1e-8, Tree="bisect")
    _, H = hm.NewHmat(hm.Params(**prm))
    x = np.random.default_rng(1).standard_normal(n)
    y = H * x
    for lo, hi in ((0, 512), (512, 2560), (3584, 4096)):
        _, S = hm.NewHmat(hm.Params(RowRange=(lo, hi), **prm))
        z = S * x
        assert np.array_equal(z[lo:hi], y[lo:hi]) and not z[:lo].any() and not z[hi:].any()
