"""The Gramians and their product with the factors (the fit gradient's W P) at
the edges of the Gramian kernel's blocks: rows around 1, 32 and 128, ranks around
1, 16 and 32, against FP64."""
import pytest
import torch

from tensorfox_gb300 import autograd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,eps", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
@pytest.mark.parametrize("dims", [(1, 2, 3), (31, 32, 33), (127, 128, 129), (160, 161, 257), (4, 3, 5, 2)])
@pytest.mark.parametrize("R", [1, 2, 3, 15, 16, 17, 33])
def test_wp1(dims, R, dtype, eps):
    g = torch.Generator(device="cuda").manual_seed(sum(dims) + R)
    W = [torch.randn((d, R), device="cuda", dtype=dtype, generator=g) for d in dims]
    W64 = [w.double() for w in W]

    def products(F):
        G, out = [f.t() @ f for f in F], []
        for l in range(len(F)):
            P = torch.ones_like(G[0])
            for m, Gm in enumerate(G):
                if m != l:
                    P = P * Gm
            out.append(F[l] @ P)
        return out

    # the Gramians' sums in FP64 of products in the working type, their product
    # rounded once, and the sum over the rank
    n = 2 * len(dims) + R + 8 + (max(dims) * len(dims) if dtype == torch.float64 else 0)
    for got, ref, mag in zip(autograd._wp1(W), products(W64), products([w.abs() for w in W64])):
        assert torch.all((got.double() - ref).abs() <= n * eps * mag)
