"""Differentiable CP layer (torch.autograd.Function) on the GB300 kernels.

* ``cp_reconstruct(factors)`` returns the dense tensor [[W_0, ..., W_{L-1}]]
  (Conversion.py:52-79 ``cpd2tens``); its backward for an incoming gradient G is
  ``dL/dW_l = MTTKRP(G, l)`` computed by ``tfx_mttkrp``.
* ``cp_fit_loss(T, factors)`` returns ``||[[W]] - T||^2`` (fused residual, the
  model is never materialised); its backward is
  ``2 (W_l P1_l - MTTKRP(T, l))`` -- twice the gradient ``g`` of
  GaussNewton.py:401-427 -- and ``2 (T - [[W]])`` for ``T`` when requested.

Both recompute the Khatri-Rao rows inside the kernels instead of storing them.
Factors are CUDA tensors of shape (d_l, R), float32 or float64.
"""
import ctypes

import torch

from . import _dev, _lib


def _vp(t):
    return t.data_ptr()


def _st():
    return _dev.stream()


def _dt(t):
    return _lib.F64 if t.dtype == torch.float64 else _lib.F32


def _cint(v):
    return (ctypes.c_int * len(v))(*v)


def _flat(factors, dtype=None):
    """The factors as one flat vector of column-major blocks, of ``dtype`` (the
    factors' own by default): one launch that reads them where they lie, whatever
    their strides (a view whose values are still to be negated goes through torch,
    which does that)."""
    W0 = factors[0]
    dt = W0.dtype if dtype is None else dtype
    L, R, dev = len(factors), W0.shape[-1], W0.device
    if (1 < L <= _lib.MAX_ORDER and dev.type == "cuda" and dt in (torch.float32, torch.float64) and
            all(W.dtype == dt and W.device == dev and W.dim() == 2 and W.shape[1] == R and W.shape[0] > 0 and R > 0 and
                not W.is_neg() for W in factors)):
        lib = _declare()
        dims = [W.shape[0] for W in factors]
        out = torch.empty(R * sum(dims), dtype=dt, device=dev)
        strides = [W.stride() for W in factors]
        _lib.check(lib.tfx_factors_pack(_lib.F64 if dt == torch.float64 else _lib.F32, L, _cint(dims), R,
                                        (ctypes.c_void_p * L)(*[W.data_ptr() for W in factors]),
                                        (ctypes.c_longlong * L)(*[s[0] for s in strides]),
                                        (ctypes.c_longlong * L)(*[s[1] for s in strides]), out.data_ptr(), _st()))
        return out
    out = torch.cat([W.detach().t().contiguous().reshape(-1) for W in factors])
    return out if dtype is None else out.to(dtype)


_DECLARED = None


def _declare():
    global _DECLARED
    if _DECLARED is not None:
        return _DECLARED
    lib = _lib.load()
    P, I, SZ = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t
    lib.tfx_mttkrp.argtypes = [I, P, I, ctypes.POINTER(ctypes.c_int), I, P, I, P, P, SZ, P]
    lib.tfx_mttkrp_scratch_bytes.restype = SZ
    lib.tfx_mttkrp_scratch_bytes.argtypes = [I, I, ctypes.POINTER(ctypes.c_int), I, I]
    lib.tfx_mttkrp_all.argtypes = [I, P, I, ctypes.POINTER(ctypes.c_int), I, P, P, I, P, SZ, P]
    lib.tfx_mttkrp_all_scratch_bytes.restype = SZ
    lib.tfx_mttkrp_all_scratch_bytes.argtypes = [I, I, ctypes.POINTER(ctypes.c_int), I]
    lib.tfx_cp_full.argtypes = [I, I, ctypes.POINTER(ctypes.c_int), I, P, P, P]
    lib.tfx_cp_wp1.argtypes = [I, I, ctypes.POINTER(ctypes.c_int), I, P, P, P, P]
    lib.tfx_cp_wp1_scratch_bytes.restype = SZ
    lib.tfx_cp_wp1_scratch_bytes.argtypes = [I, I]
    lib.tfx_factors_pack.argtypes = [I, I, ctypes.POINTER(ctypes.c_int), I, P, P, P, P, P]
    lib.tfx_cp_fit_loss.argtypes = [I, P, I, ctypes.POINTER(ctypes.c_int), I, P, P, P, P]
    lib.tfx_cp_fit_backward.argtypes = [I, P, I, ctypes.POINTER(ctypes.c_int), I, P, P, P, P, SZ, P]
    lib.tfx_cp_fit_grad.argtypes = [I, P, I, ctypes.POINTER(ctypes.c_int), I, P, P, P, SZ, P]
    lib.tfx_cp_fit_grad_scratch_bytes.restype = SZ
    lib.tfx_cp_fit_grad_scratch_bytes.argtypes = [I, I, ctypes.POINTER(ctypes.c_int), I]
    _DECLARED = lib
    return lib


def mttkrp(T, factors, mode):
    """T_(l) times the Khatri-Rao product of the other factors, as (d_l, R)."""
    lib = _declare()
    T = T.contiguous()
    dims = list(T.shape)
    L, R, dt, cd = len(dims), int(factors[0].shape[1]), _dt(T), _cint(dims)
    W = _flat(factors, T.dtype)
    nb = int(lib.tfx_mttkrp_scratch_bytes(dt, L, cd, R, int(mode)))
    scratch = torch.empty(max(nb, 16), dtype=torch.uint8, device=T.device)
    out = torch.empty((R, dims[mode]), dtype=T.dtype, device=T.device)
    _lib.check(lib.tfx_mttkrp(dt, _vp(T), L, cd, R, _vp(W), int(mode), _vp(out), _vp(scratch), nb, _st()))
    return out.t()


def _outputs(dims, R, wanted, dtype, device):
    """A contiguous (d_l, R) tensor for every wanted mode (None for the others)
    and the array of their addresses."""
    out = [torch.empty((d, R), dtype=dtype, device=device) if w else None for d, w in zip(dims, wanted)]
    return out, (ctypes.c_void_p * len(dims))(*[None if o is None else o.data_ptr() for o in out])


def mttkrp_all(T, W_flat, dims, R, wanted=None):
    """The MTTKRPs of every wanted mode, contiguous (d_l, R) tensors (one
    ``tfx_mttkrp_all`` call)."""
    lib = _declare()
    L, dt, cd = len(dims), _dt(T), _cint(dims)
    nb = int(lib.tfx_mttkrp_all_scratch_bytes(dt, L, cd, R))
    scratch = torch.empty(nb, dtype=torch.uint8, device=T.device)
    out, ptrs = _outputs(dims, R, [True] * L if wanted is None else wanted, T.dtype, T.device)
    _lib.check(lib.tfx_mttkrp_all(dt, _vp(T), L, cd, R, _vp(W_flat), ptrs, 1, _vp(scratch), nb, _st()))
    return out


def cp_full(factors):
    lib = _declare()
    dims = [int(W.shape[0]) for W in factors]
    R = int(factors[0].shape[1])
    W = _flat(factors)
    out = torch.empty(dims, dtype=W.dtype, device=W.device)
    _lib.check(lib.tfx_cp_full(_dt(W), len(dims), _cint(dims), R, _vp(W), _vp(out), _st()))
    return out


def _wp1(factors):
    lib = _declare()
    dims = [int(W.shape[0]) for W in factors]
    R = int(factors[0].shape[1])
    W = _flat(factors)
    out = torch.empty_like(W)
    scratch = torch.empty(int(lib.tfx_cp_wp1_scratch_bytes(len(dims), R)), dtype=torch.uint8, device=W.device)
    _lib.check(lib.tfx_cp_wp1(_dt(W), len(dims), _cint(dims), R, _vp(W), _vp(out), _vp(scratch), _st()))
    res, s = [], 0
    for d in dims:
        res.append(out[s:s + d * R].view(R, d).t())
        s += d * R
    return res


class CPReconstruct(torch.autograd.Function):
    @staticmethod
    def forward(ctx, *factors):
        ctx.save_for_backward(*factors)
        return cp_full(factors)

    @staticmethod
    def backward(ctx, G):
        factors = ctx.saved_tensors
        G = G.contiguous().to(factors[0].dtype)
        if sum(ctx.needs_input_grad) > 1:
            R = int(factors[0].shape[1])
            return tuple(mttkrp_all(G, _flat(factors, G.dtype), list(G.shape), R, ctx.needs_input_grad))
        return tuple(mttkrp(G, factors, l) if ctx.needs_input_grad[l] else None for l in range(len(factors)))


def fit_grad(T, W_flat, dims, R):
    """Flat gradient of ||T - [[W]]||^2: 2 (W_l P1_l - MTTKRP(T, l)) per mode
    (one ``tfx_cp_fit_grad`` call)."""
    lib = _declare()
    cd = _cint(dims)
    nb = int(lib.tfx_cp_fit_grad_scratch_bytes(_dt(T), len(dims), cd, R))
    scratch = torch.empty(nb, dtype=torch.uint8, device=T.device)
    out = torch.empty_like(W_flat)
    _lib.check(lib.tfx_cp_fit_grad(_dt(T), _vp(T), len(dims), cd, R, _vp(W_flat), _vp(out), _vp(scratch), nb, _st()))
    return out


class CPFitLoss(torch.autograd.Function):
    @staticmethod
    def forward(ctx, T, *factors):
        lib = _declare()
        T = T.contiguous()
        dims = list(T.shape)
        R = int(factors[0].shape[1])
        W_flat = _flat(factors, T.dtype)
        ctx.save_for_backward(T, W_flat, *factors)
        scratch = torch.empty(int(lib.tfx_cp_residual_scratch_bytes()), dtype=torch.uint8, device=T.device)
        loss = torch.empty((), dtype=T.dtype, device=T.device)
        _lib.check(lib.tfx_cp_fit_loss(_dt(T), _vp(T), len(dims), _cint(dims), R, _vp(W_flat), _vp(loss),
                                       _vp(scratch), _st()))
        return loss

    @staticmethod
    def backward(ctx, gl):
        T, W_flat, *factors = ctx.saved_tensors
        dims = [int(W.shape[0]) for W in factors]
        R = int(factors[0].shape[1])
        grads = [None] * len(factors)
        wanted = ctx.needs_input_grad[1:]
        if any(wanted) and torch.is_grad_enabled() and gl.requires_grad:
            # differentiated again (``create_graph``): scaled in torch, which
            # records that the gradients depend on ``gl``
            g, s = fit_grad(T, W_flat, dims, R).mul_(gl.to(T.dtype)), 0
            for l, d in enumerate(dims):
                if wanted[l]:
                    grads[l] = g[s:s + d * R].view(R, d).t().to(factors[l].dtype)
                s += d * R
        elif any(wanted):
            lib = _declare()
            L, dt, cd = len(dims), _dt(T), _cint(dims)
            nb = int(lib.tfx_cp_fit_grad_scratch_bytes(dt, L, cd, R))
            scratch = torch.empty(nb, dtype=torch.uint8, device=T.device)
            grads, ptrs = _outputs(dims, R, wanted, T.dtype, T.device)
            _lib.check(lib.tfx_cp_fit_backward(dt, _vp(T), L, cd, R, _vp(W_flat), _vp(gl.to(T.dtype)), ptrs,
                                               _vp(scratch), nb, _st()))
            grads = [None if g is None else g.to(W.dtype) for g, W in zip(grads, factors)]
        gT = 2.0 * gl * (T - cp_full(factors)) if ctx.needs_input_grad[0] else None
        return (gT, *grads)


def cp_reconstruct(factors):
    """Dense [[W_0, ..., W_{L-1}]] with an MTTKRP backward."""
    _dev.require_cuda()
    return CPReconstruct.apply(*factors)


def cp_fit_loss(T, factors):
    """||[[W]] - T||^2 with the Gauss-Newton gradient as backward."""
    _dev.require_cuda()
    return CPFitLoss.apply(T, *factors)
