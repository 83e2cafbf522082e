"""GPU: the matvec autotuner tries every phase-2 shape whatever shape the handle
is set to, BF16 factors included: row slabs are their default, and after a window
shape was set by hand the autotuner is the way back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["F64", "F32", "BF16"])
def test_slabs_are_tried_from_any_shape(storage):
    import hmatrix as hm
    n = 20011
    _, H = hm.NewHmat(hm.Params(Geom=np.sort(np.random.default_rng(1).uniform(0, 10, n)), Kernel=hm.Cauchy(1.0),
                                MaxBlock=512, MinBlock=64, MaxRank=16, ConsMethod="aca2", εComp=1e-8, Tree="bisect",
                                Storage=getattr(hm, storage)))
    x = np.random.default_rng(2).standard_normal(n)
    y = H * x                                            # row slabs: the default
    assert H.info().tune_p2_split == 1
    H.set_tune(4)
    table, choice = H.autotune(1, calls=5)
    slabs = [table["clusters_waves%d" % w] for w in (1, 2, 4)]
    assert all(v > 0 for v in slabs)
    assert (choice["p2_split"] == 1) == (min(slabs) < min(v for k, v in table.items() if k.startswith("split")))
    if choice["p2_split"] == 1:
        assert np.array_equal(H * x, y)                  # phase 1's grid does not change the sums
