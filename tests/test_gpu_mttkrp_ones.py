"""MTTKRPs and fit gradients of tensors with modes of size 1, at every place (a 1 x
1 convolution's weights, leading and trailing ones, several of them): the factors
of those modes scale the result like any other.  Against FP64."""
import itertools

import pytest
import torch

import tensorfox_gb300 as tfx

pytestmark = pytest.mark.gpu

SHAPES = [(64, 48, 1, 1), (1, 64, 48), (1, 1, 9, 7), (13, 1, 48, 1), (1, 70, 1, 5), (5, 1, 1, 1, 6), (1, 1), (1, 9),
          (9, 1), (1, 1, 1), (40, 1, 300), (1, 3, 27, 10), (5, 98, 2, 3, 1), (200, 1, 1, 150)]


@pytest.mark.parametrize("dtype,eps", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
@pytest.mark.parametrize("dims,R", list(itertools.product(SHAPES, (1, 6, 75))))
def test_modes_of_size_one(dims, R, dtype, eps):
    g = torch.Generator(device="cuda").manual_seed(sum(dims) + R)
    T = torch.randn(dims, device="cuda", dtype=dtype, generator=g)
    W = [torch.randn((d, R), device="cuda", dtype=dtype, generator=g) for d in dims]
    W64, T64, s = [w.double() for w in W], T.double(), "abcde"[:len(dims)]
    full = ",".join(c + "z" for c in s) + "->" + s

    def mttkrp(X, F, m):
        o = [i for i in range(len(dims)) if i != m]
        return torch.einsum(s + "," + ",".join(s[i] + "z" for i in o) + "->" + s[m] + "z", X, *[F[i] for i in o])

    K = T.numel()
    aW = [w.abs() for w in W64]
    leaves = [w.clone().requires_grad_(True) for w in W]
    grads = torch.autograd.grad(tfx.cp_fit_loss(T, leaves), leaves)
    back = torch.autograd.grad(tfx.cp_reconstruct(leaves), leaves, T)
    D64, aD = torch.einsum(full, *W64) - T64, torch.einsum(full, *aW) + T64.abs()
    for m, d in enumerate(dims):
        ref, mag = mttkrp(T64, W64, m), mttkrp(T64.abs(), aW, m)
        # one rounding a step at most, and the Khatri-Rao products'
        tol = (K // d + len(dims) + 4) * eps * mag
        assert torch.all((tfx.mttkrp(T, W, m).double() - ref).abs() <= tol), m
        assert torch.all((back[m].double() - ref).abs() <= tol), m
        # the gradient 2 (W P - M) from Gramians: their sums, products and the rank's besides
        gref, gmag = 2 * mttkrp(D64, W64, m), 2 * mttkrp(aD, aW, m)
        assert torch.all((grads[m].double() - gref).abs() <= (K // d + sum(dims) + R + 20) * eps * gmag), m
