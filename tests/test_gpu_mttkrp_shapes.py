"""MTTKRPs whose modes differ by orders of magnitude (a mode of thousands beside
ones of a few, Khatri-Rao blocks around the plan's limits of 8 and 64 MB, rows of a
middle mode next to a short last one), against FP64."""
import pytest
import torch

import tensorfox_gb300 as tfx

pytestmark = pytest.mark.gpu

# 8 x ldp x rows of F at 8 MB: 131072 rows of 16 columns in FP32
SHAPES = [((5, 40000, 3), 8), ((5, 43690, 3), 16), ((5, 43691, 3), 16), ((5, 150000, 7), 16), ((5, 150000, 7), 17),
          ((3, 30000, 9), 14), ((39, 51351, 4), 14), ((3, 2, 30000, 2), 5), ((2, 60000, 2, 2), 33)]


@pytest.mark.parametrize("dtype,eps", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
@pytest.mark.parametrize("dims,R", SHAPES)
def test_every_mode(dims, R, dtype, eps):
    g = torch.Generator(device="cuda").manual_seed(sum(dims) + R)
    T = torch.randn(dims, device="cuda", dtype=dtype, generator=g)
    W = [torch.randn((d, R), device="cuda", dtype=dtype, generator=g).requires_grad_(True) for d in dims]
    s = "abcd"[:len(dims)]
    with torch.no_grad():
        refs = []
        for m in range(len(dims)):
            o = [i for i in range(len(dims)) if i != m]
            eq = s + "," + ",".join(s[i] + "z" for i in o) + "->" + s[m] + "z"
            K = T.numel() // dims[m]
            F = [W[i].double() for i in o]
            ref, mag = torch.einsum(eq, T.double(), *F), torch.einsum(eq, T.double().abs(), *[f.abs() for f in F])
            refs.append(ref)
            # no chain is longer than 4096 steps, and the products' own roundings
            tol = (min(K, 4096) + len(dims) + 40) * eps * mag
            assert torch.all((tfx.mttkrp(T, W, m).double() - ref).abs() <= tol), m
    X = tfx.cp_reconstruct(W)
    for m, (got, ref) in enumerate(zip(torch.autograd.grad(X, W, T), refs)):
        assert float((got.double() - ref).norm()) <= 200 * eps * float(ref.norm()), m
