"""GPU: the dense leaves of a BF16 handle (stored in FP32) in the single-column
products: FP64 products with the FP64 vector, in both directions and in every
phase-2 shape.  One dense leaf is the whole matrix here, cut into one slab, or
into several with a short last one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# FP64 sums of exact products of the stored FP32 entries
@pytest.mark.parametrize("n", [5, 33, 64, 301, 1000])
def test_bf16_dense_leaves(n):
    import hmatrix as hm
    rng = np.random.default_rng(n)
    _, H = hm.NewHmat(hm.Params(Geom=np.sort(rng.uniform(0, 10, n)), Kernel=hm.Cauchy(1.0), MaxBlock=n, MinBlock=n,
                                MaxRank=8, ConsMethod="aca2", εComp=1e-9, Tree="bisect", Storage=hm.BF16))
    D = H.to_dense()
    x = rng.standard_normal(n)
    for split in (None, 4):                        # the default (row slabs), windows
        if split:
            H.set_tune(split)
        for A, trans in ((D, False), (D.T, True)):
            y = H.matvec(x, trans=trans)
            assert np.abs(y - A @ x).max() <= 8 * n * 2.0 ** -53 * (np.abs(A) @ np.abs(x)).max()
