"""The sparse MTTKRP and residual over the lane splits of their FP32 forms (R 4,
8, 12 and up in fours, other ranks), orders two to five, entry counts that are
no multiple of a warp's share, factor rows off a 16-byte boundary, and both ways
of passing the factors' addresses, against FP64 sums on the host."""
import ctypes

import numpy as np
import pytest
import torch

from tensorfox_gb300 import _lib, sparse

pytestmark = pytest.mark.gpu

U = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53}


def data(dims, nnz, R, dtype, shift):
    rng = np.random.RandomState(nnz + R)
    idx = np.stack([rng.randint(0, d, nnz) for d in dims], axis=1)
    vals = rng.randn(nnz)
    X = sparse.DeviceCOO(vals.astype(np.float32 if dtype == torch.float32 else np.float64), idx, dims, dtype)
    W = []
    for d in dims:
        buf = torch.from_numpy(rng.randn(d * R + 1)).to("cuda", dtype)
        W.append(buf[1:].view(d, R) if shift else buf[:-1].view(d, R))
    v = X.vals.double().cpu().numpy()
    w = [a.double().cpu().numpy() for a in W]
    return X, W, idx, v, w


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dims,nnz,R,shift", [((7, 5, 6), 1, 4, False), ((40, 30, 20), 1001, 4, False),
                                              ((40, 30, 20), 1003, 8, False), ((40, 30, 20), 997, 12, True),
                                              ((9, 30, 20), 4099, 20, False), ((40, 30, 20), 999, 5, False),
                                              ((11, 9, 8, 7), 515, 8, False), ((11, 9, 8, 7), 513, 16, True),
                                              ((6, 5, 4, 3, 7), 301, 4, False), ((50, 60), 333, 24, False)])
def test_products_and_residual(dims, nnz, R, shift, dtype):
    X, W, idx, v, w = data(dims, nnz, R, dtype, shift)
    L, u = len(dims), U[dtype]
    rows = [w[m][idx[:, m]] for m in range(L)]
    for mode in range(L):
        p = np.ones((nnz, R)) * v[:, None]
        for m in range(L):
            if m != mode:
                p = p * rows[m]
        ref, mag = np.zeros((dims[mode], R)), np.zeros((dims[mode], R))
        np.add.at(ref, idx[:, mode], p)
        np.add.at(mag, idx[:, mode], np.abs(p))
        # L products an entry; float-float (or FP64: at most nnz) additions, one final rounding
        tol = (L + 2 + (nnz if dtype == torch.float64 else 0)) * u
        got = sparse.coo_mttkrp(X, W, mode).double().cpu().numpy()
        assert np.all(np.abs(got - ref) <= tol * mag + 1e-300)
    model, mag = np.prod(rows, axis=0).sum(axis=1), np.abs(np.prod(rows, axis=0)).sum(axis=1)
    ref = np.sum((v - model) ** 2)
    # an entry's model carries at most L + R roundings, the difference one
    d = (L + R + 2) * u * (mag + np.abs(v))
    tol = np.sum(2 * np.abs(v - model) * d + d * d) + (nnz * 2.0 ** -53 + 1e-13) * ref
    got = float(sparse.sparse_residual_sq(X, W)[0])
    assert abs(got - ref) <= tol
    # addresses in a device array: the same kernels, the same sums
    ptrs = sparse._row_major_ptrs(W)
    out = torch.empty((dims[0], R), dtype=dtype, device="cuda")
    rowptr, sidx, svals = X.sort_mode(0)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _lib.call("tfx_coo_mttkrp", X.dt(), vp(sidx), vp(svals), X.nnz, vp(rowptr), L, sparse._cint(dims), R, 0,
              vp(ptrs), vp(out), st)
    assert torch.equal(out, sparse.coo_mttkrp(X, W, 0))


def test_missing_row_is_refused():
    X, W, *_ = data((4, 5, 6), 10, 4, torch.float32, False)
    rowptr, sidx, svals = X.sort_mode(0)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    ptrs = (ctypes.c_void_p * 3)(W[0].data_ptr(), None, W[2].data_ptr())
    out = torch.empty((4, 4), dtype=torch.float32, device="cuda")
    with pytest.raises(_lib.TfxError):
        _lib.call("tfx_coo_mttkrp_rows", X.dt(), vp(sidx), vp(svals), X.nnz, vp(rowptr), 3, sparse._cint((4, 5, 6)),
                  4, 0, ptrs, vp(out), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
