"""The work that is measured: what a program that uses this package has it do.

An H-matrix is built once on a cluster tree and then multiplied by vectors (in
both directions, one column or a block of them, with FP64, FP32 or BF16
factors), factorised, solved with, and differentiated through; many small
independent systems come as one batch.  The configurations are those of the
package's benchmark and tests (the 1-D Cauchy matrix on [0, 10], the 2-D point
cloud, the Gaussian kernel of the gradient leg, the uneven batch) with their
block sizes and tolerances, at sizes from the README's n = 2000 to n = 2^19,
powers of two and ragged ones.

``listed`` names the cases, ``draw`` gives more of the same ranges; ``prepare``
makes what a program has in hand before the call, ``run`` is one pass through
the public entry points, ``work`` the bytes and operations it cannot do
without, and ``exact`` the same results from dense FP64 arithmetic.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "hmatrix.jl_b200"))
import hmatrix as hm  # noqa: E402

STORAGE = {"f64": hm.F64, "f32": hm.F32, "bf16": hm.BF16}


# -- cases -------------------------------------------------------------------
def _matvec(n, **kw):
    """The 1-D benchmark matrix: 1/(1+(x-y)^2/l^2) on [0, 10], MaxBlock 512."""
    c = dict(kind="matvec", n=n, dim=1, points="grid", tree="bisect", kernel="cauchy", p=1.0, shift=0.0,
             max_block=512, min_block=64, max_rank=16, tol=1e-8, cons="aca2", storage="f64", ncols=1, trans=False)
    c.update(kw)
    return c


def _cloud(n, **kw):
    """The 2-D point cloud of the benchmark: uniform in [0,1]^2, 1/(1+|x-y|^2) + 1e-3 I."""
    return _matvec(n, **dict(dict(dim=2, points="random", shift=1e-3, max_rank=32, tol=1e-9), **kw))


def _lu(n, **kw):
    """The H-LU leg: 1/(1+(x-y)^2) + delta_xy, MaxBlock 256, MinBlock 32, MaxRank 12."""
    return _matvec(n, **dict(dict(kind="lu", shift=1.0, max_block=256, min_block=32, max_rank=12, tol=1e-10,
                                  eps_lu=0.0), **kw))


def _gradient(n, **kw):
    """The differentiation leg: exp(-(x-y)^2/(2 l^2)) + s^2 I, l = 0.7, s^2 = 1e-2."""
    return _matvec(n, **dict(dict(kind="gradient", kernel="gauss", p=0.7, shift=1e-2, max_rank=24, tol=1e-10), **kw))


def _batch(count, nmin, nmax, **kw):
    """The uneven batch: n log-uniform, sorted uniform points on [0, L], L ~ U[5, 20], l ~ U[0.5, 2]."""
    return _lu(nmax, **dict(dict(kind="batch", count=count, nmin=nmin, points="random", pick=1), **kw))


def listed():
    return [
        # the README's program: 2000 points, the KMeans tree, SVD compression;
        # one product as a Krylov loop calls it (launches and latency)
        dict(_matvec(2000, tree="kmeans", max_block=500, max_rank=5, tol=1e-10, cons="svd"), name="matvec_readme_n2000"),
        # scattered 1-D points, a size that no tree divides evenly
        dict(_matvec(100003, points="random", p=0.8), name="matvec_1d_ragged"),
        # the largest FP64 product: streams the factors from HBM
        dict(_matvec(2 ** 19), name="matvec_1d_large"),
        # H'x of a 2-D point cloud (adjoint products, both halves of BiCG-like solvers)
        dict(_cloud(70001, trans=True), name="matvec_2d_adjoint"),
        # FP32 factors inside a single-precision program (vectors in and out in FP32)
        dict(_matvec(300000, storage="f32"), name="matvec_f32"),
        # block of right-hand sides in FP64 (block Krylov, several responses at once)
        dict(_matvec(2 ** 17, kind="block", ncols=16), name="block16_f64"),
        # the same with FP32 factors
        dict(_matvec(200000, kind="block", ncols=16, storage="f32"), name="block16_f32"),
        # many probing vectors with BF16 factors, adjoint direction
        dict(_matvec(2 ** 18, kind="block", ncols=64, storage="bf16", trans=True), name="block64_bf16_adjoint"),
        # construction: a program whose geometry or kernel changes each step
        # compresses the matrix anew, then multiplies by it
        dict(_cloud(50000, kind="build"), name="build_2d"),
        # factorise and solve to a relative residual of 1e-10
        dict(_lu(2 ** 16), name="lu_solve"),
        # forward and backward of b'(H\b) + |Hb|^2 through stored factors (hyper-parameter fits)
        dict(_gradient(20000), name="gradient"),
        # many small independent systems, factorised and solved in one call
        dict(_batch(16, 2 ** 10, 2 ** 13, eps_lu=1e-6), name="batch_lu_solve"),
    ]


def _size(rng, lo, hi):
    """Log-uniform in [lo, hi]; one in four a power of two, the others as they fall."""
    n = int(round(2.0 ** rng.uniform(math.log2(lo), math.log2(hi))))
    if rng.random() < 0.25:
        n = max(1 << (n.bit_length() - 1), 1)
        n = n if n >= lo else 2 * n
    return min(n, hi)


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "matvec", "cloud", "block", "block", "build", "lu", "gradient", "batch"])
    p = round(rng.uniform(0.5, 2.0), 6)
    points = rng.choice(["grid", "random"])
    trans = rng.random() < 0.4
    if kind == "matvec":
        storage = rng.choice(["f64", "f64", "f32", "bf16"])
        return _matvec(_size(rng, 2000, 2 ** 19), p=p, points=points, trans=trans, storage=storage)
    if kind == "cloud":
        return _cloud(_size(rng, 4000, 100000), p=p, trans=trans)
    if kind == "block":
        storage = rng.choice(["f64", "f32", "bf16"])
        return _matvec(_size(rng, 4000, 2 ** 17 if storage == "f64" else 2 ** 18), kind="block", p=p, points=points,
                       trans=trans, storage=storage, ncols=rng.choice([2, 3, 8, 16, 24, 32, 64]))
    if kind == "build":
        if rng.random() < 0.5:
            return _cloud(_size(rng, 4000, 50000), kind="build", p=p)
        return _matvec(_size(rng, 4000, 2 ** 17), kind="build", p=p, points=points)
    if kind == "lu":
        return _lu(_size(rng, 2 ** 11, 2 ** 15), p=p, points=points, eps_lu=rng.choice([0.0, 1e-6]),
                   ncols=rng.choice([1, 1, 8]))
    if kind == "gradient":
        return _gradient(_size(rng, 4000, 20000), p=round(rng.uniform(0.5, 1.0), 6), points=points)
    return _batch(rng.choice([4, 8, 16]), 2 ** 10, 2 ** 13, eps_lu=rng.choice([0.0, 1e-6]),
                  pick=rng.randrange(2, 10 ** 6))


# -- inputs --------------------------------------------------------------------
def _points(case, rng, n, length=10.0):
    if case["dim"] == 2:
        return rng.uniform(0.0, 1.0, (n, 2))
    if case["points"] == "grid":
        return np.linspace(0.0, length, n)
    return np.sort(rng.uniform(0.0, length, n))


def _params(case, geom, p=None, **kw):
    kernel = {"cauchy": hm.Cauchy, "gauss": hm.Gauss}[case["kernel"]](case["p"] if p is None else p)
    return hm.Params(Geom=geom, Kernel=kernel, MaxBlock=case["max_block"], MinBlock=case["min_block"],
                     MaxRank=case["max_rank"], ConsMethod=case["cons"], εComp=case["tol"], Tree=case["tree"],
                     Storage=STORAGE[case["storage"]], Shift=case["shift"], εTruncLU=case.get("eps_lu", 0.0), **kw)


def _inputs(case, seed):
    """(geometry, right-hand sides) of one system, from the seed alone."""
    rng = np.random.default_rng(seed)
    geom = _points(case, rng, case["n"])
    shape = case["n"] if case["ncols"] == 1 else (case["n"], case["ncols"])
    return geom, rng.standard_normal(shape)


def _batch_inputs(case, seed):
    """[(geometry, l, right-hand side)] of a batch, from the seed alone; the sizes are the case's own."""
    sizes = np.random.default_rng(case["pick"])
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        n = int(round(2.0 ** sizes.uniform(math.log2(case["nmin"]), math.log2(case["n"]))))
        geom = _points(case, rng, n, length=rng.uniform(5.0, 20.0))
        out.append((geom, rng.uniform(0.5, 2.0), rng.standard_normal(n)))
    return out


def _single(case):
    """Reduced factors sit in a single-precision program: its vectors are FP32."""
    return case["storage"] != "f64"


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        probs = _batch_inputs(case, seed)
        return {"case": case, "H": [hm.NewHmat(_params(case, g, p))[1] for g, p, _ in probs], "y": [y for _, _, y in probs]}
    geom, x = _inputs(case, seed)
    state = {"case": case}
    if kind == "gradient":
        op = hm_operator(_params(case, geom))
        op.L, op.dH                                       # the factors a training loop holds
        state.update(op=op, b=torch.tensor(x, device="cuda", requires_grad=True))
    elif kind == "build":
        c = hm.construct_cluster(geom if geom.ndim == 2 else geom.reshape(-1, 1), case["min_block"], case["tree"])
        state.update(prm=_params(case, geom), c=c, x=torch.tensor(x, device="cuda"))
    elif kind == "lu":
        state.update(H=hm.NewHmat(_params(case, geom))[1], y=x)
    else:
        c, H = hm.NewHmat(_params(case, geom))
        state.update(H=H, x=torch.tensor(x, device="cuda", dtype=torch.float32 if _single(case) else torch.float64))
    return state


def hm_operator(prm):
    from hmatrix.autodiff import KernelOperator
    return KernelOperator(prm, refine_tol=1e-13)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("matvec", "block"):
        if _single(case):
            return state["H"].matvec(state["x"].double(), trans=case["trans"]).float()
        return state["H"].matvec(state["x"], trans=case["trans"])
    if kind == "build":
        return hm.new_on_cluster(state["prm"], state["c"]).matvec(state["x"])
    if kind == "lu":
        return hm.lu(state["H"]).solve_refined(state["y"], tol=1e-10, max_iter=20)[0]
    if kind == "gradient":
        op, b = state["op"], state["b"]
        loss = torch.dot(b, op.solve(b)) + torch.sum(op.matvec(b) ** 2)
        gb, gp, gs = torch.autograd.grad(loss, [b, op.p, op.sigma2])
        return {"loss": loss.detach(), "b": gb, "p": gp, "sigma2": gs}
    Ls = hm.lu_batch(state["H"])
    return hm.solve_refined_batch(Ls, state["y"], tol=1e-10, max_iter=20)[0]


# -- what a pass cannot do without ----------------------------------------------
def _lu_flops(n, case, rank):
    """Recompressions of the T^3/3 trailing updates of T tiles of MaxBlock rows
    (a QR of both stacked factors of 2 rank columns and the new factors:
    6 (m + n) (2 rank)^2 each)."""
    s = min(case["max_block"], n)
    t = max(1.0, n / s)
    return t ** 3 / 3.0 * 6.0 * (2 * s) * (2 * rank) ** 2 + t * 2.0 / 3.0 * s ** 3


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = {"bytes": 0, "flops": 0}
        for geom, p, y in _batch_inputs(case, 0):
            o = hm.NewHmat(_params(case, geom, p))[1].info()
            rank = o.rk_entries / max(1, o.n_rk) / (2.0 * case["max_block"])
            total["bytes"] += 2 * o.pool_bytes + 16 * len(y)
            total["flops"] += _lu_flops(len(y), case, max(1.0, rank))
        return total
    geom, _ = _inputs(case, 0)
    o = hm.NewHmat(_params(case, geom))[1].info()
    vec = (4 if _single(case) else 8) * 2 * case["n"] * case["ncols"]
    factors = o.matvec_bytes - 16 * case["n"]
    entries = o.rk_entries + o.dense_entries
    if kind in ("matvec", "block"):
        return {"bytes": factors + vec, "flops": 2 * entries * case["ncols"]}
    rank = max(1.0, o.rk_entries / max(1, o.n_rk) / (2.0 * case["max_block"]))
    if kind == "build":
        # kernel values of every stored entry (about 8 operations), the cross
        # approximation's updates, and the factors written and read once
        return {"bytes": 2 * factors + vec, "flops": entries * (8 + 2 * rank) + 2 * entries}
    if kind == "lu":
        return {"bytes": 2 * o.pool_bytes + vec, "flops": _lu_flops(case["n"], case, rank)}
    # gradient: two refined solves (two sweeps over the LU factors each, here
    # counted as the size of H) and four products
    return {"bytes": 8 * factors + 10 * vec, "flops": 16 * entries}


# -- dense FP64 values -------------------------------------------------------------
class _Dense:
    """Products with the dense kernel matrix on the GPU, FP64, a slab of rows at a time."""

    def __init__(self, case, geom, p=None, deriv=False):
        X = np.asarray(geom, dtype=np.float64)
        self.X = torch.tensor(X.reshape(len(X), -1), device="cuda")
        self.kernel, self.p, self.deriv = case["kernel"], case["p"] if p is None else p, deriv
        self.shift = 0.0 if deriv else case["shift"]
        self.rows = max(1, min(len(X), 8 * 1024 * 1024 // len(X)))     # a slab stays in L2
        self.buf = torch.empty((2, self.rows, len(X)), dtype=torch.float64, device="cuda")

    def __call__(self, v):
        X, n = self.X, len(self.X)
        v2 = v.reshape(n, -1)
        out = self.shift * v2
        for r in range(0, n, self.rows):
            e = min(n, r + self.rows)
            s, t = self.buf[0, :e - r], self.buf[1, :e - r]
            torch.sub(X[r:e, 0, None], X[None, :, 0], out=s)
            s.mul_(s)
            for q in range(1, X.shape[1]):
                torch.sub(X[r:e, q, None], X[None, :, q], out=t)
                s.addcmul_(t, t)
            if self.kernel == "cauchy":
                s.div_(self.p * self.p).add_(1.0).reciprocal_()
            elif self.deriv:
                torch.mul(s, 1.0 / self.p ** 3, out=t)
                s.div_(-2.0 * self.p * self.p).exp_().mul_(t)
            else:
                s.div_(-2.0 * self.p * self.p).exp_()
            out[r:e] += s @ v2
        return out.reshape(v.shape)


def _cg(A, b):
    """A x = b for the symmetric positive definite A, to rounding (each column by itself)."""
    cols = []
    for y in b.reshape(len(b), -1).t():
        y = y.contiguous()
        x = torch.zeros_like(y)
        for _ in range(2):                                 # the second round works on the true residual
            r = y - A(x)
            d, rr = r.clone(), torch.dot(r, r)
            x0, tol = torch.zeros_like(y), 1e-15 * float(torch.linalg.norm(r))
            for _ in range(400):
                if float(rr) ** 0.5 <= tol:
                    break
                q = A(d)
                a = rr / torch.dot(d, q)
                x0 += a * d
                r -= a * q
                new = torch.dot(r, r)
                d = r + (new / rr) * d
                rr = new
            x = x + x0
        cols.append(x)
    return torch.stack(cols, 1).reshape(b.shape)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for geom, p, y in _batch_inputs(case, seed):
            out.append(_cg(_Dense(case, geom, p), torch.tensor(y, device="cuda")))
        return out
    if case["n"] > 2 ** 19 or (kind == "lu" and case["n"] * case["ncols"] > 2 ** 16):
        return None
    geom, x = _inputs(case, seed)
    x = torch.tensor(x, device="cuda")
    if kind != "gradient" and case["dim"] == 2:
        geom = geom[hm.construct_cluster(geom, case["min_block"], case["tree"]).P]
    elif case["tree"] == "kmeans":
        geom = geom[hm.construct_cluster(geom.reshape(-1, 1), case["min_block"], case["tree"]).P]
    A = _Dense(case, geom)
    if kind in ("matvec", "block"):
        return A(x.float().double() if _single(case) else x)   # the kernel is symmetric
    if kind == "build":
        return A(x)
    if kind == "lu":
        return _cg(A, x)
    dA = _Dense(case, geom, deriv=True)
    s, h = _cg(A, x), A(x)
    ds, dh = dA(s), dA(x)
    return {"loss": torch.dot(x, s) + torch.dot(h, h), "b": 2 * s + 2 * A(h),
            "p": -torch.dot(s, ds) + 2 * torch.dot(h, dh), "sigma2": -torch.dot(s, s) + 2 * torch.dot(h, x)}
