"""Performance cases of the framework: what its users have it do, through its
public functions.

A case is a dict of plain values.  ``listed()`` gives the fixed ones and
``draw(rng)`` one more of the same ranges; ``prepare`` makes a case's inputs and
what a program keeps beside them, ``run`` is one pass, ``work`` the bytes and
operations such a pass cannot do without, and ``exact`` the same results in 64
bits by plain torch.

Kinds of case, and what each stands for in use:

* ``fit``: one training step's loss and gradients of a CP model against a dense
  tensor (``cp_fit_loss`` and its backward): convolution weights being
  factorised, and data tensors of order 3 and 4;
* ``reconstruct``: a CP-parametrised tensor inside a larger differentiable
  program (``cp_reconstruct``), forward and backward from an upstream gradient;
* ``mttkrp``: the products of one sweep over the modes (an alternating or a
  gradient method of the user's own), ``mttkrp`` for every mode;
* ``compress``: the sequential truncation of a dense tensor with known bases,
  the Gram of every mode and the mode products, in each of the three precisions
  that ``cpd`` takes;
* ``coo``: the products of one sweep and the residual on a sparse tensor;
* ``dgn``: the damped Gauss-Newton solver on a compressed core from a start the
  caller has, a fixed number of iterations;
* ``cpd``: the whole decomposition with default options.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensor-fox_gb300"))

import tensorfox_gb300 as tfx  # noqa: E402
from tensorfox_gb300 import kernels  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # a 3 x 3 convolution layer's weights at rank 64, the repository's own
        # differentiation workload: short modes, bound by launches and latency
        dict(name="fit_256x256x3x3_r64_f32", kind="fit", dims="256,256,3,3", rank=64, dtype="f32"),
        # a data tensor of ordinary, odd sizes
        dict(name="fit_187x143x95_r21_f32", kind="fit", dims="187,143,95", rank=21, dtype="f32"),
        # the benchmark's full tensor, larger than the L2
        dict(name="fit_512x512x512_r50_f32", kind="fit", dims="512,512,512", rank=50, dtype="f32"),
        # double precision, fourth order, no mode a multiple of a tile
        dict(name="fit_45x38x31x26_r12_f64", kind="fit", dims="45,38,31,26", rank=12, dtype="f64"),
        # a CP layer of a larger model: the dense tensor out, its gradient in
        dict(name="reconstruct_300x262x217_r40_f32", kind="reconstruct", dims="300,262,217", rank=40, dtype="f32"),
        # one sweep of an alternating method
        dict(name="mttkrp_384x320x256_r48_f32", kind="mttkrp", dims="384,320,256", rank=48, dtype="f32"),
        # the benchmark's compression (precision 'mixed')
        dict(name="compress_512x512x512_n50_mixed", kind="compress", dims="512,512,512", rank=50, dtype="mixed"),
        # the default precision of float32 and of float64 input
        dict(name="compress_384x320x256_n40_f32", kind="compress", dims="384,320,256", rank=40, dtype="f32"),
        dict(name="compress_150x141x130_n20_f64", kind="compress", dims="150,141,130", rank=20, dtype="f64"),
        # the sparse workload of the benchmark: 20000^3, 1e7 stored entries
        dict(name="coo_20000x20000x20000_1e7_r16_f32", kind="coo", dims="20000,20000,20000", nnz=10_000_000, rank=16,
             dtype="f32"),
        # the benchmark's compressed core
        dict(name="dgn_50x50x50_r50_f32", kind="dgn", dims="50,50,50", rank=50, dtype="f32"),
        # the plain double-precision decomposition, default options
        dict(name="cpd_100x100x100_r10_f64", kind="cpd", dims="100,100,100", rank=10, dtype="f64"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _text(dims):
    return ",".join(str(int(d)) for d in dims)


def _dense_dims(rng, order, entries, least=6):
    """``order`` mode sizes whose product is at most ``entries``, each at most
    about six times the geometric mean."""
    total = entries ** (1.0 / order)
    d = [max(least, int(total * 6.0 ** (rng.random() - 0.5))) for _ in range(order)]
    while np.prod([float(v) for v in d]) > entries:
        d[d.index(max(d))] -= max(1, max(d) // 16)
    return d


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "reconstruct", "mttkrp", "mttkrp", "compress", "compress", "coo", "dgn",
                       "cpd"])
    if kind in ("fit", "reconstruct", "mttkrp"):
        dtype = "f64" if rng.random() < 0.25 else "f32"
        top = 3e6 if dtype == "f64" else 6e7
        if kind == "fit" and rng.random() < 0.3:
            k = rng.choice([3, 5, 7])
            dims = [_log_int(rng, 32, 512), _log_int(rng, 32, 512), k, k]
            return dict(kind=kind, dims=_text(dims), rank=_log_int(rng, 8, 64), dtype=dtype)
        order = rng.choice([3, 3, 3, 4, 5])
        dims = _dense_dims(rng, order, float(_log_int(rng, 20_000, int(top))))
        return dict(kind=kind, dims=_text(dims), rank=_log_int(rng, 3, 64), dtype=dtype)
    if kind == "compress":
        dtype = rng.choice(["mixed", "f32", "f64"])
        top = {"mixed": 9e7, "f32": 3e7, "f64": 3e6}[dtype]
        dims = _dense_dims(rng, rng.choice([3, 3, 4]), float(_log_int(rng, 60_000, int(top))), least=12)
        return dict(kind=kind, dims=_text(dims), rank=min(_log_int(rng, 4, 60), min(dims)), dtype=dtype)
    if kind == "coo":
        order = rng.choice([3, 3, 4])
        dims = [_log_int(rng, 300, 20_000) for _ in range(order)]
        dtype = "f64" if rng.random() < 0.25 else "f32"
        return dict(kind=kind, dims=_text(dims), nnz=_log_int(rng, 10_000, 5_000_000), rank=_log_int(rng, 3, 32),
                    dtype=dtype)
    if kind == "dgn":
        dims = [rng.randint(12, 56) for _ in range(3)]
        return dict(kind=kind, dims=_text(dims), rank=min(_log_int(rng, 4, 50), min(dims)), dtype="f32")
    dims = [rng.randint(30, 110) for _ in range(3)]
    return dict(kind=kind, dims=_text(dims), rank=rng.randint(3, 10), dtype="f64")


def _dims(case):
    return [int(d) for d in case["dims"].split(",")]


def _dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _letters(order):
    return "abcdefgh"[:order]


def _model(W):
    """The dense tensor of the factors by plain torch, in their type."""
    rest = W[-1]
    for w in reversed(W[1:-1]):
        rest = (w[:, None, :] * rest[None, :, :]).reshape(-1, w.shape[1])
    return (W[0] @ rest.t()).reshape([w.shape[0] for w in W])


def _planted(dims, rank, g, noise, dtype=torch.float32):
    """Gaussian factors with entries near unit scale and the tensor they make,
    with Gaussian noise of ``noise`` times its norm."""
    W = [torch.randn((d, rank), device=DEV, generator=g, dtype=dtype) for d in dims]
    T = _model(W)
    E = torch.randn(dims, device=DEV, generator=g, dtype=dtype)
    T = T + (noise * T.norm() / E.norm()) * E
    return T, W


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    dims, rank, dt, kind = _dims(case), int(case["rank"]), _dtype(case), case["kind"]
    st = dict(kind=kind, dims=dims, rank=rank)
    if kind in ("fit", "mttkrp"):
        # a tensor with structure and 10% noise; factors half way to it
        T, W = _planted(dims, rank, g, 0.1, dt)
        W = [w + 0.5 * torch.randn(w.shape, device=DEV, generator=g, dtype=dt) for w in W]
        st["T"] = T.contiguous()
        st["W"] = [w.requires_grad_() for w in W] if kind == "fit" else W
    elif kind == "reconstruct":
        st["W"] = [torch.randn((d, rank), device=DEV, generator=g, dtype=dt).requires_grad_() for d in dims]
        st["G"] = torch.randn(dims, device=DEV, generator=g, dtype=dt)
    elif kind == "compress":
        T, W = _planted(dims, rank, g, 0.01, dt)
        st["T"] = T.contiguous()
        # bases as a program keeps them: orthonormal rows, (n, d) contiguous
        st["U"] = [torch.linalg.qr(w)[0].t().contiguous() for w in W]
        st["tc"] = case["dtype"] == "mixed"
    elif kind == "coo":
        nnz = int(case["nnz"])
        idx = torch.stack([torch.randint(0, d, (nnz,), device=DEV, generator=g) for d in dims], 1)
        W = [torch.randn((d, rank), device=DEV, generator=g, dtype=dt) for d in dims]
        vals = torch.ones((nnz, rank), device=DEV, dtype=dt)
        for l in range(len(dims)):
            vals *= W[l][idx[:, l]]
        vals = vals.sum(1)
        vals += 0.01 * vals.std() * torch.randn(nnz, device=DEV, generator=g, dtype=dt)
        st["X"] = tfx.DeviceCOO(vals.cpu().numpy(), idx.cpu().numpy(), dims, dt)
        # factors off the planted ones, as they are in mid-solve
        st["W"] = [(w + 0.3 * torch.randn(w.shape, device=DEV, generator=g, dtype=dt)).contiguous() for w in W]
    elif kind == "dgn":
        T, W = _planted(dims, rank, g, 0.01, dt)
        st["T"] = T.contiguous()
        start = [w + 0.3 * torch.randn(w.shape, device=DEV, generator=g, dtype=dt) for w in W]
        st["start"] = [w.double().cpu().numpy() for w in start]
        o = tfx.make_options(False)
        o.maxiter = 6
        st["options"] = o
    else:
        T, _ = _planted(dims, rank, g, 1e-4, torch.float64)
        st["T"] = T.contiguous()
        st["options"] = tfx.make_options(False)
    st["seed"] = int(seed) % (1 << 31)
    return st


def run(st):
    kind = st["kind"]
    if kind == "fit":
        for w in st["W"]:
            w.grad = None
        loss = tfx.cp_fit_loss(st["T"], st["W"])
        loss.backward()
        return [loss.detach()] + [w.grad for w in st["W"]]
    if kind == "reconstruct":
        for w in st["W"]:
            w.grad = None
        X = tfx.cp_reconstruct(st["W"])
        X.backward(st["G"])
        return [X.detach()] + [w.grad for w in st["W"]]
    if kind == "mttkrp":
        return [tfx.mttkrp(st["T"], st["W"], l) for l in range(len(st["W"]))]
    if kind == "compress":
        S, shape, tc = st["T"], list(st["dims"]), st["tc"]
        grams, flags = [], []
        for l, U in enumerate(st["U"]):
            if tc and kernels.tc_gram_supported(S, shape, l):
                G, flag = kernels.mode_gram_tc(S, shape, l, check=False)
                flags.append(flag)
            else:
                G = kernels.mode_gram(S, shape, l)
            grams.append(G)
            S, shape = kernels.ttm(S, shape, l, U, tensor_cores=tc)
        if tc:                       # the kernels' error flags, as a program reads them
            for flag in flags:
                kernels.check_gram_flag(flag)
            kernels.check_ttm_flag()
        return grams + [S]
    if kind == "coo":
        X, W = st["X"], st["W"]
        out = [tfx.coo_mttkrp(X, W, l) for l in range(len(W))]
        # the residual in the data's own type: that is what it is computed in
        return out + [tfx.sparse_residual_sq(X, W).to(X.vals.dtype)]
    np.random.seed(st["seed"])       # the solver draws its CG caps and its start from NumPy
    if kind == "dgn":
        W, _, errors, _, _, _ = tfx.dGN(st["T"], [w.copy() for w in st["start"]], st["rank"], st["options"])
        # a float32 solve: its results in the type it is computed in
        return [w.astype(np.float32) for w in W] + [np.asarray(errors, dtype=np.float32)]
    W, out = tfx.cpd(st["T"], st["rank"], st["options"])
    return list(W) + [float(out.rel_error)]


def work(case):
    dims, R, kind = _dims(case), int(case["rank"]), case["kind"]
    L, N, S = len(dims), float(np.prod([float(d) for d in dims])), float(sum(dims))
    s = 8 if case["dtype"] == "f64" else 4
    if kind == "fit":
        # the tensor read forward and backward, factors in and gradients out;
        # the model and, backward, the products of all modes by a dimension
        # tree (two contractions of the whole tensor)
        return dict(bytes=2 * N * s + 3 * S * R * s, flops=6 * N * R)
    if kind == "reconstruct":
        return dict(bytes=2 * N * s + 3 * S * R * s, flops=6 * N * R)
    if kind == "mttkrp":
        return dict(bytes=N * s + 2 * S * R * s, flops=4 * N * R)
    if kind == "compress":
        cur, nb, fl = list(dims), N * s, 0.0
        for l in range(L):
            n = float(np.prod([float(d) for d in cur]))
            fl += n * (cur[l] + 1) + 2 * n * R           # half of the symmetric Gram; the product
            nb += cur[l] * cur[l] * s + R * cur[l] * s
            cur[l] = R
        return dict(bytes=nb + float(R) ** L * s, flops=fl)
    if kind == "coo":
        nnz = float(case["nnz"])
        return dict(bytes=(L + 1) * nnz * (4 * L + s) + (2 * L + 1) * S * R * s, flops=(2 * L * L + 2 * L + 2) * nnz * R)
    if kind == "dgn":
        # six iterations of gradient (dimension tree) and error; each CG step is
        # a few R x R products of the factors
        return dict(bytes=N * s + 3 * S * R * s, flops=6 * 6 * N * R)
    n = [float(min(R, d)) for d in dims]
    return dict(bytes=2 * N * s + 2 * S * R * s, flops=N * (dims[0] + 1) + 2 * N * n[0] + 2 * N * R)


def _mttkrp64(T, W, l):
    """T_(l) times the Khatri-Rao product of the other factors, in 64 bits, a
    column at a time so that nothing of the tensor's size is made twice."""
    L, cols = len(W), []
    for r in range(W[0].shape[1]):
        x = T
        for m in range(L - 1, l, -1):
            x = x @ W[m][:, r]
        for m in range(l):
            x = torch.tensordot(W[m][:, r], x, dims=([0], [0]))
        cols.append(x)
    return torch.stack(cols, 1)


def _gram64(T, l):
    M = T.movedim(l, 0).reshape(T.shape[l], -1)
    return M @ M.t()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("dgn", "cpd"):
        return None                  # iterates, not values that 64 bits give
    st = prepare(case, seed)
    if kind == "coo":
        X, W = st["X"], [w.double() for w in st["W"]]
        vals, idx = X.vals.double(), X.idx32.long()
        L, R = len(W), W[0].shape[1]
        out = [torch.zeros((d, R), device=DEV, dtype=torch.float64) for d in st["dims"]]
        res = torch.zeros(1, device=DEV, dtype=torch.float64)
        for b in range(0, vals.numel(), 1 << 20):
            v, ix = vals[b:b + (1 << 20)], idx[:, b:b + (1 << 20)]
            rows = [W[m][ix[m]] for m in range(L)]
            for l in range(L):
                p = v[:, None].expand(-1, R).clone()
                for m in range(L):
                    if m != l:
                        p *= rows[m]
                out[l].index_add_(0, ix[l], p)
            model = rows[0].clone()
            for m in range(1, L):
                model *= rows[m]
            res += ((v - model.sum(1)) ** 2).sum()
        return out + [res]
    if kind == "compress":
        S, out = st["T"].double(), []
        for l, U in enumerate(st["U"]):
            out.append(_gram64(S, l))
            S = torch.tensordot(U.double(), S, dims=([1], [l])).movedim(0, l)
        return out + [S.contiguous()]
    W = [w.detach().double() for w in st["W"]]
    if kind == "reconstruct":
        G = st["G"].double()
        return [_model(W)] + [_mttkrp64(G, W, l) for l in range(len(W))]
    T = st["T"].double()
    if kind == "mttkrp":
        return [_mttkrp64(T, W, l) for l in range(len(W))]
    E = T - _model(W)
    loss = (E * E).sum()
    return [loss] + [-2.0 * _mttkrp64(E, W, l) for l in range(len(W))]
