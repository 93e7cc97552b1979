"""The engine's third-order gradient, J^T J products and residual at the edges
of their tiles (16, 32 and 64 rows and columns, odd and even extents, ranks on
either side of the rule that shares out slabs or columns, one CTA and more than
there are slabs), against the same quantities in FP64 on the host."""
import numpy as np
import pytest
import torch

import tensorfox_gb300 as tfx
from tensorfox_gb300 import _dev, _lib
from tensorfox_gb300 import gauss_newton as gn

pytestmark = pytest.mark.gpu

U = {"fp32": 2.0 ** -24, "fp64": 2.0 ** -53}


def problem(dims, R, precision):
    rng = np.random.RandomState(sum(dims) * 100 + R)
    dt = np.float32 if precision == "fp32" else np.float64
    W = [rng.randn(d, R).astype(dt) for d in dims]
    T = (np.einsum("ir,jr,kr->ijk", *[w.astype(np.float64) for w in W]) + rng.randn(*dims)).astype(dt)
    v = rng.randn(sum(dims) * R).astype(dt)
    return T, W, v


def products(T, W, v):
    """gradient W_l P1_l - M_l and J^T J v (flat, modes in order, columns contiguous)"""
    dims, R = T.shape, W[0].shape[1]
    G = [w.T @ w for w in W]
    D, o = [], 0
    for d in dims:
        D.append(v[o:o + d * R].reshape(R, d).T)
        o += d * R
    M = [np.einsum("ijk,jr,kr->ir", T, W[1], W[2]), np.einsum("ijk,ir,kr->jr", T, W[0], W[2]),
         np.einsum("ijk,ir,jr->kr", T, W[0], W[1])]
    P1 = [G[1] * G[2], G[0] * G[2], G[0] * G[1]]
    grad = [W[l] @ P1[l] - M[l] for l in range(3)]
    A = [D[k].T @ W[k] for k in range(3)]
    jv = []
    for l in range(3):
        Y = sum(G[3 - l - k] * A[k] for k in range(3) if k != l)
        jv.append(W[l] @ Y + D[l] @ P1[l])
    flat = lambda x: np.concatenate([m.T.ravel() for m in x])  # noqa: E731
    return flat(grad), flat(jv), M


SIZES = [((16, 16, 16), 16), ((3, 17, 5), 16), ((9, 16, 16), 17), ((5, 32, 32), 32), ((6, 33, 31), 20),
         ((4, 64, 64), 64), ((7, 64, 2), 3), ((64, 2, 64), 33), ((13, 15, 12), 1), ((2, 4, 8), 64),
         ((5, 60, 56), 65), ((50, 50, 50), 50), ((10, 10, 10), 10)]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dims,R", SIZES)
def test_gradient_and_product(dims, R, precision):
    T, W, v = problem(dims, R, precision)
    t, w, x = T.astype(np.float64), [a.astype(np.float64) for a in W], v.astype(np.float64)
    g, jv, _ = products(t, w, x)
    # every term of either product passes through at most this many roundings
    # (three contractions over extents, one over the rank, the products between)
    n = sum(dims) + 2 * R + 32
    aw, av = [np.abs(a) for a in w], np.abs(x)
    _, bj, bm = products(np.abs(t), aw, av)
    bg = np.concatenate([(bm[l] + aw[l] @ P).T.ravel() for l, P in enumerate(
        [(aw[1].T @ aw[1]) * (aw[2].T @ aw[2]), (aw[0].T @ aw[0]) * (aw[2].T @ aw[2]),
         (aw[0].T @ aw[0]) * (aw[1].T @ aw[1])])])
    tol = 2 * n * U[precision]
    ran = 0
    for cluster in sorted({1, min(2, R), min(16, R)}):
        try:
            got_g, got_j = gn.jtj_matvec(T, W, R, v=v, damp=0.0, cluster=cluster, precision=precision)
        except _lib.TfxError as e:  # a plan above the shared memory is refused
            assert "use a larger cluster" in str(e) and R >= 33
            continue
        ran += 1
        eg = np.abs(got_g.double().cpu().numpy() - g)
        ej = np.abs(got_j.double().cpu().numpy() - jv)
        assert np.all(eg <= tol * bg), (cluster, np.max(eg / bg) / U[precision], n)
        assert np.all(ej <= tol * bj), (cluster, np.max(ej / bj) / U[precision], n)
    assert ran or precision == "fp64"


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dims,R,cluster", [((16, 16, 16), 4, 1), ((9, 33, 31), 5, 2), ((11, 32, 32), 6, 4),
                                            ((5, 36, 50), 8, 8), ((10, 10, 10), 10, 8), ((3, 4, 64), 2, 2)])
def test_solve_reports_the_error_of_its_factors(dims, R, cluster, precision):
    T, W, _ = problem(dims, R, precision)
    o = tfx.make_options(False)
    o.maxiter = 4
    x0 = torch.from_numpy(_dev.flat_factors([w.astype(np.float64) for w in W])).to("cuda", _dev.torch_dtype(precision))
    b = gn.dGN_device(torch.from_numpy(T).cuda(), x0, R, o, precision, cluster=cluster)
    x = b.best[0].double().cpu().numpy()
    F, p = [], 0
    for d in dims:
        F.append(x[p:p + d * R].reshape(R, d).T)
        p += d * R
    t = T.astype(np.float64)
    err = np.linalg.norm(t - np.einsum("ir,jr,kr->ijk", *F)) / np.linalg.norm(t)
    model = np.linalg.norm(np.einsum("ir,jr,kr->ijk", *[np.abs(f) for f in F])) / np.linalg.norm(t)
    got = float(b.info[0, 1])
    # the model's entries carry R + 3 roundings, the sums of squares less than 1e-6 of their value
    assert abs(got - err) <= (R + 8) * U[precision] * model + (1e-6 if precision == "fp32" else 1e-13) * err
