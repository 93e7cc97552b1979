"""The FP32 model kernel (``cp_fit_loss`` forward, ``cpd2tens``) at the edges of
its tiles, against the model in FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows around 8 and 64, columns around 128 and 256 and odd ones, ranks around 4
# and 64, one mode of size 1, orders 2 to 5, several row tiles a block
SHAPES = [((3, 5, 7), 1), ((8, 16, 8), 4), ((9, 127), 5), ((64, 128), 3), ((65, 129), 64), ((66, 13, 21), 65),
          ((7, 300, 3, 3), 130), ((200, 257), 9), ((12, 9, 8, 7, 6), 6), ((300, 40, 1), 20), ((40, 700, 130), 12)]


@pytest.mark.parametrize("dims,R", SHAPES)
def test_model_and_residual(dims, R):
    import tensorfox_gb300 as tfx
    g = torch.Generator(device="cuda").manual_seed(sum(dims) + R)
    W = [torch.randn((d, R), device="cuda", generator=g) for d in dims]
    s = "abcde"[:len(dims)]
    eq = ",".join(c + "r" for c in s) + "->" + s
    ref = torch.einsum(eq, *[w.double() for w in W])
    mag = torch.einsum(eq, *[w.double().abs() for w in W])
    X = tfx.cpd2tens(W)
    # a product's L - 1 roundings and at most R of the sum
    n = R + len(dims) + 2
    assert torch.all((X.double() - ref).abs() <= n * 2.0 ** -24 * mag + 1e-30)
    for shift in (0, 1):   # one element off the 16-byte boundary
        T = torch.randn(int(np.prod(dims)) + shift, device="cuda", generator=g)[shift:].view(dims)
        loss = tfx.cp_fit_loss(T, W)
        d = T.double() - ref
        # the model's error and the difference's own rounding, to first order
        # and squared, and the rounding of the result
        e = n * 2.0 ** -24 * mag + 2.0 ** -24 * d.abs()
        tol = (2 * d.abs() * e + e * e).sum() + 2.0 ** -23 * (d * d).sum()
        assert abs(float(loss) - float((d * d).sum())) <= float(tol), shift
