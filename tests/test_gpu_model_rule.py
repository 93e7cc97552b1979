"""FP32 model and residual on both sides of the rule that picks between 64 x 64
tiles and the register-tiled kernel (leading mode, rank and number of elements at
the line, leading modes of one to a few rows), against the model in FP64."""
import pytest
import torch

import tensorfox_gb300 as tfx

pytestmark = pytest.mark.gpu

SHAPES = [((3, 3, 256, 256), 64), ((8, 1000, 130), 8), ((31, 180, 180), 8), ((32, 180, 180), 8), ((14, 71431), 2),
          ((64, 217, 217), 9), ((65, 217, 217), 9), ((65, 46154), 64), ((66, 20, 30, 80), 64), ((66, 20, 30, 80), 65),
          ((1, 9), 1), ((100000, 31), 64), ((2, 1, 1), 130)]


@pytest.mark.parametrize("dims,R", SHAPES)
def test_model_and_residual(dims, R):
    g = torch.Generator(device="cuda").manual_seed(sum(dims) + R)
    W = [torch.randn((d, R), device="cuda", generator=g) for d in dims]
    s = "abcd"[:len(dims)]
    eq = ",".join(c + "r" for c in s) + "->" + s
    ref = torch.einsum(eq, *[w.double() for w in W])
    mag = torch.einsum(eq, *[w.double().abs() for w in W])
    # a product's L - 1 roundings and at most R of the sum
    n = R + len(dims) + 2
    assert torch.all((tfx.cpd2tens(W).double() - ref).abs() <= n * 2.0 ** -24 * mag + 1e-30)
    T = torch.randn(dims, device="cuda", generator=g)
    loss = float(tfx.cp_fit_loss(T, W))
    d = T.double() - ref
    # the model's error and the difference's own rounding, to first order and
    # squared, and the rounding of the result
    e = n * 2.0 ** -24 * mag + 2.0 ** -24 * d.abs()
    tol = (2 * d.abs() * e + e * e).sum() + 2.0 ** -23 * (d * d).sum()
    assert abs(loss - float((d * d).sum())) <= float(tol)
