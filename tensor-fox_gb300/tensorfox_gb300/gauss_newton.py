"""Damped Gauss-Newton on the device (GaussNewton.py:29 ``dGN``).

``dGN(T, factors, R, options)`` keeps the reference's signature and return
tuple.  The whole iteration (CG inner solves, dogleg fallback, damping updates
and stop tests) runs as one launch of the cluster-persistent engine
(``tfx_dgn_solve``); the host only prepares the CG caps and reads the results.

The 'cg' inner method draws its CG cap from NumPy's global RNG once per
iteration (GaussNewton.py:267).  The caps are drawn here from a copy of the RNG
state, and afterwards the real RNG is advanced by exactly the draws the
reference would have made, so seeded runs stay in step with it.
"""
import ctypes

import numpy as np
import torch

from . import _dev, _lib
from .options import make_options


def _inner_of(options, it):
    im = options.inner_method
    return im[it] if isinstance(im, list) else im


def cg_budgets(options, L):
    """CG caps for every iteration, drawn without consuming the global RNG."""
    state = np.random.get_state()
    out = np.zeros(options.maxiter, dtype=np.int32)
    try:
        for it in range(options.maxiter):
            inner = _inner_of(options, it)
            if inner == 'cg':
                out[it] = 1 + (L - 2) * int(options.cg_factor * np.random.randint(1 + it ** 0.4, 2 + it ** 0.9))
            elif inner == 'cg_static':
                out[it] = options.cg_maxiter
            else:
                raise NotImplementedError(
                    "inner_method %r is outside the damped Gauss-Newton CG path" % (inner,))
    finally:
        np.random.set_state(state)
    return out


def advance_rng(options, iterations):
    """Consumes the RNG draws the reference's 'cg' caps make in ``iterations`` steps."""
    for it in range(iterations):
        if _inner_of(options, it) == 'cg':
            np.random.randint(1 + it ** 0.4, 2 + it ** 0.9)


def auto_cluster(dims, R, problems=1):
    """CTAs per problem (one thread-block cluster): at most R, since every CTA
    owns whole factor columns, and 16, or 8 where the core has fewer than 1e5
    multiply-adds a product (the step from 8 to 16 then gains nothing).  One
    CTA's own SM bounds small problems, in FP64 by its FP64 pipe.  Ten
    iterations, one CTA against the cluster chosen: 10^3 R 10 FP64 3.8 -> 1.6 ms,
    FP32 1.04 -> 0.71; 30^3 R 30 FP64 28.7 -> 3.7, FP32 4.3 -> 0.96 (two CTAs:
    15.8 and 2.4); 4^3 R 4 FP32 0.65 -> 0.64.  ``problems`` solved in one launch
    share the GPU's 152 SMs: no more CTAs than those, but about one CTA per 1.2
    million multiply-adds of per-iteration MTTKRP work.  It knows nothing of solves
    in flight on other streams: a program that keeps the GPU full of small ones
    sets ``options.cluster`` (one CTA is the least SM time)."""
    n = int(np.prod(dims))
    alone = 16 if n * R >= 100000 else 8
    share = max(152 // problems, n * R * len(dims) // 1200000)
    return int(max(1, min(16, R, alone, share)))


def _cluster_candidates(c, R, auto=False):
    """Cluster sizes to try in turn: ``c``, then wider ones, whose CTAs need less
    shared memory, and for a size that ``auto_cluster`` chose (``auto``) also
    narrower ones, for a device that cannot schedule that many CTAs together."""
    R = max(R, 1)
    if auto:
        c = max(1, min(c, R))
    cands = [c] + [x for x in (1, 2, 4, 8, 12, 16) if x > c]
    if auto:
        cands += [x for x in (12, 8, 4, 2, 1) if x < c]
    return [x for x in cands if x <= R] or [1]


def _first_that_fits(cands, launch):
    """The first size that ``launch`` does not refuse as unsupported."""
    for c in cands:
        status = launch(c)
        if status != 5:
            break
    _lib.check(status)
    return c


class _Batch:
    """Device buffers for a set of dGN problems solved in one engine launch."""

    def __init__(self, tensors, xs, R_list, options, precision, budgets=None, aliased=False, fix_mode=-1):
        self.precision = precision
        dt = _dev.torch_dtype(precision)
        self.es = 8 if precision == "fp64" else 4
        lib = _lib.load()
        self.n = len(tensors)
        self.options = options
        self.maxiter = int(options.maxiter)
        self.tensors = tensors
        self.xs = xs
        self.dims = [tuple(int(d) for d in t.shape) for t in tensors]
        self.R = R_list
        self.best = [torch.empty_like(x) for x in xs]
        self.ws = []
        for t, R in zip(tensors, R_list):
            L = t.dim()
            dims_c = (ctypes.c_int * L)(*t.shape)
            nb = lib.tfx_dgn_workspace_bytes(_dev.lib_dtype(precision), L, dims_c, int(R))
            self.ws.append(torch.empty(int(nb), dtype=torch.uint8, device=t.device))
        # One pinned block holds the descriptors (the library copies them to the
        # device itself), the CG caps and the damping schedule; the latter two go
        # over in one asynchronous copy, queued behind the device work.  One
        # zeroed device block takes what the engine reports.  This object keeps
        # both alive until the results are read.
        dev = tensors[0].device
        if budgets is None:
            budgets = [cg_budgets(options, t.dim()) for t in tensors]
        caps = np.concatenate([np.asarray(b, dtype=np.int32) for b in budgets])
        sched = options.init_damp if isinstance(options.init_damp, list) else None
        sc = np.asarray(sched if sched is not None else [], dtype=np.float64)
        nd = ctypes.sizeof(_lib.DgnProblem) * self.n
        o_sc = (nd + 15) // 16 * 16
        o_cap = o_sc + 8 * sc.size
        self._host = torch.empty(o_cap + 4 * caps.size, dtype=torch.uint8, pin_memory=True)
        view = self._host.numpy()
        view[:nd] = 0
        view[o_sc:o_cap].view(np.float64)[:] = sc
        view[o_cap:].view(np.int32)[:] = caps
        self.d_desc = torch.empty(self._host.numel(), dtype=torch.uint8, device=dev)
        self.d_desc[o_sc:].copy_(self._host[o_sc:], non_blocking=True)
        base = self.d_desc.data_ptr()
        caps_at = base + o_cap + 4 * np.concatenate([[0], np.cumsum([len(b) for b in budgets])])
        self.sched = sched
        n, m = self.n, self.maxiter
        self._out = torch.zeros(n * (2 + 4 * m + 8 + 24), dtype=torch.float64, device=dev)
        self.result = self._out[:2 * n].view(torch.int32).view(n, 4)
        self.stats = self._out[2 * n:n * (2 + 4 * m)].view(n, 4 * m)
        self.info = self._out[n * (2 + 4 * m):n * (10 + 4 * m)].view(n, 8)
        self.prof = self._out[n * (10 + 4 * m):].view(torch.int64).view(n, 24)
        self.desc = (_lib.DgnProblem * self.n).from_address(self._host.data_ptr())
        for p in range(self.n):
            d = self.desc[p]
            d.L = len(self.dims[p])
            d.R = int(R_list[p])
            for l, v in enumerate(self.dims[p]):
                d.dims[l] = v
            d.tensor = _dev.ptr(tensors[p])
            d.x = _dev.ptr(xs[p])
            d.best = _dev.ptr(self.best[p])
            d.work = _dev.ptr(self.ws[p])
            d.budgets = int(caps_at[p])
            d.damp_sched = base + o_sc if sched is not None else None
            d.stats = _dev.ptr(self.stats[p])
            d.result = _dev.ptr(self.result[p])
            d.info = _dev.ptr(self.info[p])
            d.prof = _dev.ptr(self.prof[p])
        o = _lib.DgnOptions()
        o.maxiter = self.maxiter
        o.tol, o.tol_step, o.tol_improv = float(options.tol), float(options.tol_step), float(options.tol_improv)
        o.tol_grad, o.tol_jump, o.cg_tol = float(options.tol_grad), float(options.tol_jump), float(options.cg_tol)
        o.init_damp = 0.0 if sched is not None else float(options.init_damp)
        o.use_damp_sched = 1 if sched is not None else 0
        o.symm = 1 if options.symm else 0
        o.factors_norm = float(options.factors_norm)
        o.tile = int(getattr(options, 'tile', None) or 0)
        o.aliased = 1 if aliased else 0
        o.fixed = int(fix_mode) + 1
        self.opts = o

    def report(self):
        """(result (n, 4), stats (n, 4 maxiter)) on the host, one transfer."""
        n = self.n
        h = self._out[:n * (2 + 4 * self.maxiter)].cpu().numpy()
        return h[:2 * n].view(np.int32).reshape(n, 4), h[2 * n:].reshape(n, -1)

    def launch(self, cluster, stream=None, auto=False):
        """``auto``: ``cluster`` is auto_cluster's choice, not the caller's."""
        lib = _lib.load()
        st = _dev.stream() if stream is None else stream
        return _first_that_fits(
            _cluster_candidates(cluster, min(self.R), auto),
            lambda c: lib.tfx_dgn_solve(_dev.lib_dtype(self.precision), self.desc,
                                        ctypes.c_void_p(_dev.ptr(self.d_desc)), self.n, ctypes.byref(self.opts), c,
                                        ctypes.c_void_p(st)))


def _precision_of(T, options):
    p = getattr(options, 'precision', None)
    if p in ('fp64', 'fp32'):
        return p
    if p == 'mixed':
        return 'fp32'
    if p not in (None, 'auto'):
        raise ValueError("precision must be 'fp64', 'fp32', 'mixed' or None")
    if isinstance(T, torch.Tensor):
        return 'fp64' if T.dtype == torch.float64 else 'fp32'
    return 'fp64' if np.asarray(T).dtype == np.float64 else 'fp32'


def dGN_device(Td, x0d, R, options, precision, cluster=None, aliased=False, fix_mode=-1):
    """Runs the engine on device-resident inputs; returns device results."""
    b = _Batch([Td], [x0d], [R], options, precision, aliased=aliased, fix_mode=fix_mode)
    c = cluster if cluster is not None else options.cluster
    b.launch(c or auto_cluster(Td.shape, R), auto=not c)
    return b


class _Single:
    """One problem's descriptor and workspace for the standalone evaluations."""

    def __init__(self, T, x_flat, R, precision):
        self.precision = precision
        self.dt = _dev.torch_dtype(precision)
        self.Td = _dev.to_device(T, self.dt)
        self.dims = tuple(int(d) for d in self.Td.shape)
        dev = self.Td.device
        self.x = (x_flat if isinstance(x_flat, torch.Tensor) else torch.from_numpy(np.asarray(x_flat)))
        self.x = self.x.to(dev, self.dt).contiguous()
        lib = _lib.load()
        L = len(self.dims)
        dims_c = (ctypes.c_int * L)(*self.dims)
        self.ws = torch.empty(int(lib.tfx_dgn_workspace_bytes(_dev.lib_dtype(precision), L, dims_c, int(R))),
                              dtype=torch.uint8, device=dev)
        self.result = torch.zeros(4, dtype=torch.int32, device=dev)
        d = _lib.DgnProblem()
        d.L, d.R = L, int(R)
        for l, v in enumerate(self.dims):
            d.dims[l] = v
        d.tensor, d.x, d.work, d.result = _dev.ptr(self.Td), _dev.ptr(self.x), _dev.ptr(self.ws), _dev.ptr(self.result)
        self.desc = d
        self.d_desc = torch.empty(ctypes.sizeof(_lib.DgnProblem), dtype=torch.uint8, device=dev)
        o = _lib.DgnOptions()
        o.maxiter = 1
        self.opts = o

    def vec(self, v):
        t = v if isinstance(v, torch.Tensor) else torch.from_numpy(np.ascontiguousarray(v))
        return t.to(self.Td.device, self.dt).contiguous()

    def check(self):
        _lib.check_solve_status(self.result.cpu().numpy())


def _vp(t):
    return ctypes.c_void_p(_dev.ptr(t) if t is not None else None)


def _single_candidates(cluster, dims, R):
    if cluster is not None:
        return [int(cluster)]
    return _cluster_candidates(auto_cluster(dims, R), int(R), auto=True)


def jtj_matvec(T, factors, R, v=None, damp=1.0, cluster=None, precision=None, gradient=True):
    """The solver's per-iteration products at one point, computed by the same
    device code as the solve (``tfx_jtj_matvec``): the gradient ``g`` of
    GaussNewton.py:401-427 (``compute_grad``) and ``J^T J v`` of
    GaussNewton.py:551-581 (``matvec``), both in the flat layout.

    ``T`` and ``v`` may be NumPy arrays or torch tensors; the results are
    device tensors of the working precision (``None`` for a skipped product)."""
    _dev.require_cuda()
    if precision is None:
        precision = 'fp64' if (getattr(T, 'dtype', None) in (np.float64, torch.float64)) else 'fp32'
    s = _Single(T, _dev.flat_factors(list(factors)), R, precision)
    vd = s.vec(v) if v is not None else None
    jv = torch.empty_like(s.x) if v is not None else None
    g = torch.empty_like(s.x) if gradient else None
    lib = _lib.load()
    _first_that_fits(_single_candidates(cluster, s.dims, R), lambda c: lib.tfx_jtj_matvec(
        _dev.lib_dtype(precision), ctypes.byref(s.desc), _vp(s.d_desc), ctypes.byref(s.opts), c, float(damp), _vp(vd),
        _vp(jv), _vp(g), ctypes.c_void_p(_dev.stream())))
    s.check()
    return g, jv


def dogleg_steps(T, x, y, grad, jtj, error, damp, R, cluster=None, precision=None, symm=False, factors_norm=0):
    """The dogleg trials after a rejected step (GaussNewton.py:713-795
    ``compute_dogleg_steps``) on the device, by the solver's own code.  Returns
    ``(best_factors_flat, best_x, best_y, best_error)`` as device tensors and a
    float."""
    _dev.require_cuda()
    if precision is None:
        precision = 'fp64' if (getattr(T, 'dtype', None) in (np.float64, torch.float64)) else 'fp32'
    s = _Single(T, x, R, precision)
    s.opts.symm = 1 if symm else 0
    s.opts.factors_norm = float(factors_norm)
    yd, gd, jd = s.vec(y), s.vec(grad), s.vec(jtj)
    bx, by, bw = torch.empty_like(s.x), torch.empty_like(s.x), torch.empty_like(s.x)
    be = torch.empty(1, dtype=torch.float64, device=s.x.device)
    lib = _lib.load()
    _first_that_fits(_single_candidates(cluster, s.dims, R), lambda c: lib.tfx_dgn_dogleg(
        _dev.lib_dtype(precision), ctypes.byref(s.desc), _vp(s.d_desc), ctypes.byref(s.opts), c, float(damp),
        float(error), _vp(yd), _vp(gd), _vp(jd), _vp(bx), _vp(by), _vp(bw), _vp(be), ctypes.c_void_p(_dev.stream())))
    s.check()
    return bw, bx, by, float(be.item())


def dGN(T, factors, R, options=None, precision=None):
    """Damped Gauss-Newton (GaussNewton.py:29-251) on the device.

    Returns ``(best_factors, step_sizes, errors, improv, gradients, stop)`` with
    NumPy float64 arrays, exactly like the reference.
    """
    _dev.require_cuda()
    options = make_options(options) if not hasattr(options, 'bi_method_parameters') else options
    if precision is not None:
        options.precision = precision
    prec = _precision_of(T, options)
    dt = _dev.torch_dtype(prec)
    Td = _dev.to_device(T, dt)
    dims = tuple(Td.shape)
    factors = list(factors)
    L = len(factors)
    aliased = L > 1 and all(f is factors[0] for f in factors)   # one array L times (symmetric start)
    fix = -1
    for l in range(L):        # [W] marks a fixed factor (bicpd), GaussNewton.py:92-99
        if isinstance(factors[l], list):
            fix, factors[l] = l, factors[l][0]
    x0 = _dev.h2d(_dev.flat_factors(factors), dt, Td.device)
    from .stepped import uses_stepped, dgn_stepped
    if uses_stepped(options):
        best, ss, er, im, gr, st = dgn_stepped(Td, x0, R, options, prec, fix_mode=fix, aliased=aliased)
        return (_dev.unflat(best.double().cpu().numpy(), dims, R), ss, er, im, gr, st)
    if aliased and len(set(dims)) != 1:
        raise ValueError("one factor array for every mode needs equal dimensions")
    b = dGN_device(Td, x0, R, options, prec, aliased=aliased, fix_mode=fix)
    res, stats = (v[0] for v in b.report())
    _lib.check_solve_status(res)
    n = int(res[1])
    advance_rng(options, n)
    best = _dev.unflat(b.best[0].cpu().numpy(), dims, R)
    m = options.maxiter
    return (best, stats[m:m + n].copy(), stats[:n].copy(), stats[2 * m:2 * m + n].copy(),
            stats[3 * m:3 * m + n].copy(), int(res[0]))
