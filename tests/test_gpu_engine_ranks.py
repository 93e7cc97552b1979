"""The engine's third-order relative error at ranks on both sides of 32 and 64
(the columns of one factor row that a warp's lanes hold) and well above, in both
precisions and both forms of the FP64 loop (single entries, 4 x 4 blocks), on one
CTA and on clusters, against the error of the reported factors in FP64 on the
host; and the dogleg's trials above rank 64 against the oracle."""
import numpy as np
import pytest
import torch

import tensorfox_gb300 as tfx
import tfx_oracle as orc
from tensorfox_gb300 import _dev, _lib
from tensorfox_gb300 import gauss_newton as gn

pytestmark = pytest.mark.gpu

U = {"fp32": 2.0 ** -24, "fp64": 2.0 ** -53}


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dims", [(20, 20, 20), (9, 36, 30)])
@pytest.mark.parametrize("R", [32, 33, 63, 64, 65, 70, 97, 100])
def test_error_of_the_reported_factors(dims, R, precision):
    rng = np.random.RandomState(sum(dims) * 100 + R)
    dt = np.float32 if precision == "fp32" else np.float64
    W = [rng.randn(d, R) for d in dims]
    # some noise: an error of zero would say nothing about its relative accuracy
    T = (np.einsum("ir,jr,kr->ijk", *W) + 3 * rng.randn(*dims)).astype(dt)
    o = tfx.make_options(False)
    o.maxiter = 2
    x0 = torch.from_numpy(_dev.flat_factors(W)).to("cuda", _dev.torch_dtype(precision))
    ran = 0
    for cluster in (1, 2, 16):
        try:
            b = gn.dGN_device(torch.from_numpy(T).cuda(), x0, R, o, precision, cluster=cluster)
        except _lib.TfxError as e:  # a plan above the shared memory is refused
            assert "use a larger cluster" in str(e) or "shared memory" in str(e)
            continue
        ran += 1
        x = b.best[0].double().cpu().numpy()
        F, p = [], 0
        for d in dims:
            F.append(x[p:p + d * R].reshape(R, d).T)
            p += d * R
        t = T.astype(np.float64)
        err = np.linalg.norm(t - np.einsum("ir,jr,kr->ijk", *F)) / np.linalg.norm(t)
        model = np.linalg.norm(np.einsum("ir,jr,kr->ijk", *[np.abs(f) for f in F])) / np.linalg.norm(t)
        # the model's entries carry R + 3 roundings, the sums of squares less than 1e-6 of their value
        tol = (R + 8) * U[precision] * model + (1e-6 if precision == "fp32" else 1e-13) * err
        assert abs(float(b.info[0, 1]) - err) <= tol, (cluster, float(b.info[0, 1]), err)
    assert ran


@pytest.mark.parametrize("dims,R,cluster", [((12, 10, 10), 66, 4), ((9, 36, 30), 80, 16)])
def test_dogleg_above_64(dims, R, cluster):
    rng = np.random.default_rng(R)
    W = [rng.standard_normal((d, R)) for d in dims]
    T = orc.cpd2tens(W) + 0.05 * rng.standard_normal(dims)
    n = R * sum(dims)
    x = orc.cpd2flat(W) + 0.05 * rng.standard_normal(n)
    y = 3.0 * rng.standard_normal(n)
    g2 = rng.standard_normal(n)
    j2 = 50 * g2 + rng.standard_normal(n)
    size = np.linalg.norm(T)
    err = np.linalg.norm(T - orc.cpd2tens(orc.x2cpd(x + y, [w.copy() for w in W]))) / size
    _, ref_x, ref_y, ref_e = orc.compute_dogleg_steps(size, orc.unfold(T, 1), [np.zeros((d, R)) for d in dims], g2, j2,
                                                      x.copy(), y.copy(), err, 0.3, False, 0)
    _, bx, by, be = gn.dogleg_steps(T, x, y, g2, j2, err, 0.3, R, cluster=cluster, precision="fp64")
    np.testing.assert_allclose(be, ref_e, rtol=1e-9)
    np.testing.assert_allclose(bx.cpu().numpy(), ref_x, rtol=1e-9, atol=1e-11)
    np.testing.assert_allclose(by.cpu().numpy(), ref_y, rtol=1e-9, atol=1e-11)
