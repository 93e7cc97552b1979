"""The sum of a residual's or a norm's block partials: few of them (one warp) and
many (one CTA), with one and with two values each, against FP64."""
import pytest
import torch

from tensorfox_gb300 import kernels

pytestmark = pytest.mark.gpu


# 256 elements a block of the norms, up to several hundred blocks
@pytest.mark.parametrize("n", [1, 300, 32 * 256, 33 * 256, 128 * 256, 128 * 256 + 1, 200000, 3000000])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_norms(n, dtype):
    x = torch.randn(n, device="cuda", dtype=dtype, generator=torch.Generator(device="cuda").manual_seed(n))
    got, ref = kernels.tensor_norms(x), torch.stack([(x.double() ** 2).sum(), x.double().abs().sum()])
    eps = 2.0 ** -53 if dtype == torch.float64 else 2.0 ** -24
    assert torch.all((got - ref).abs() <= 40 * eps * ref)


# one 64 x 64 tile a block: 1, 32, 33, 128, 129 and more partials
@pytest.mark.parametrize("rows", [5, 64 * 32, 64 * 32 + 1, 64 * 128, 64 * 128 + 1, 64 * 700])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_residual(rows, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows)
    W = [torch.randn((d, 2), device="cuda", dtype=dtype, generator=g) for d in (rows, 6)]
    T = torch.randn((rows, 6), device="cuda", dtype=dtype, generator=g)
    flat = torch.cat([w.t().reshape(-1) for w in W])
    got = float(kernels.cp_residual_sq(T, [rows, 6], flat, 2)[0])
    d = T.double() - W[0].double() @ W[1].double().t()
    eps = 2.0 ** -53 if dtype == torch.float64 else 2.0 ** -24
    mag = T.double().abs() + (W[0].double().abs() @ W[1].double().abs().t())
    # three roundings in a difference, and those of the sum of squares
    assert abs(got - float((d * d).sum())) <= float((8 * eps * d.abs() * mag).sum()) + 40 * eps * float((d * d).sum())
