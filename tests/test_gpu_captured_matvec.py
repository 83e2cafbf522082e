"""GPU: a single-column product may be captured into a CUDA graph once the handle
has run one in either direction: what a direction's first call would still have to
allocate (its row slab lists) is not needed for it.  The captured product replays
with the contents its input then has."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the captured call takes the window lists: the same products in another order
TOL = {"F64": 1e-14, "F32": 4e-6}


@pytest.mark.parametrize("storage", ["F64", "F32"])
def test_capture_of_the_other_direction(storage):
    import torch
    import hmatrix as hm
    n = 4096
    _, H = hm.NewHmat(hm.Params(Geom=np.linspace(0, 10, n), Kernel=hm.Cauchy(1.0), MaxBlock=512, MinBlock=64, MaxRank=16,
                                ConsMethod="aca2", εComp=1e-8, Tree="bisect", Storage=getattr(hm, storage)))
    x = torch.randn(n, device="cuda", dtype=torch.float64)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        H.matvec(x)
    torch.cuda.current_stream().wait_stream(s)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = H.matvec(x, trans=True)
    for _ in range(2):
        x.copy_(torch.randn(n, device="cuda", dtype=torch.float64))
        g.replay()
        torch.cuda.synchronize()
        z = H.matvec(x, trans=True)                      # builds the lists: row slabs from here on
        assert float(torch.linalg.norm(y - z)) <= TOL[storage] * float(torch.linalg.norm(z))
