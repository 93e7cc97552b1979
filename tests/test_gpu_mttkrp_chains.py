"""Accuracy of FP32 MTTKRPs of short modes over long contractions: rounding errors
no larger than those of chains of 128 additions.  Against FP64, in the 2-norm: a
chain of c additions of independent terms is off by sqrt(c / 2) roundings of
2^-24 / sqrt(3) in the mean square, relative to the terms' root sum of squares."""
import pytest
import torch

import tensorfox_gb300 as tfx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,R,mode", [((10, 200000, 3), 8, 2), ((3, 10, 200000), 8, 1), ((22, 22620, 13), 19, 2),
                                         ((5, 52, 8, 828), 6, 0), ((9, 410, 1360), 1, 0), ((10, 200000, 3), 8, 0),
                                         ((40, 100000, 5), 20, 2)])
def test_error_of_short_modes(dims, R, mode):
    g = torch.Generator(device="cuda").manual_seed(sum(dims) + R)
    T = torch.randn(dims, device="cuda", generator=g)
    W = [torch.randn((d, R), device="cuda", generator=g) for d in dims]
    s = "abcd"[:len(dims)]
    o = [i for i in range(len(dims)) if i != mode]
    eq = s + "," + ",".join(s[i] + "z" for i in o) + "->" + s[mode] + "z"
    ref = torch.einsum(eq, T.double(), *[W[i].double() for i in o])
    terms = torch.einsum(eq, T.double() ** 2, *[W[i].double() ** 2 for i in o]).sum().sqrt()
    err = float((tfx.mttkrp(T, W, mode).double() - ref).norm() / terms)
    assert err <= (128 / 2) ** 0.5 * 2.0 ** -24 / 3 ** 0.5
