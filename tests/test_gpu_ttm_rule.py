"""Mode products on both sides of the rules that pick a kernel by how well the
tiles fill the GPU (few and many tiles, one element off the 16-byte boundary, few
and many rows of U^T), against FP64."""
import pytest
import torch

from tensorfox_gb300 import kernels

pytestmark = pytest.mark.gpu

F32 = [(3, 394, 202, 6), (1, 33, 5001, 64), (50, 31, 129, 10), (50, 33, 129, 3), (60, 31, 128, 3), (61, 33, 128, 9),
       (31, 64, 128, 40), (31, 65, 128, 40), (152, 33, 128, 1), (151, 33, 128, 1), (100, 20, 128, 84), (400, 13, 128, 70)]


def check(P, D, Q, n, dtype, eps, shift):
    g = torch.Generator(device="cuda").manual_seed(P + 3 * D + 7 * Q + n)
    S = torch.randn(P * D * Q + shift, device="cuda", generator=g, dtype=dtype)[shift:].view(P, D, Q)
    U = torch.randn((n, D), device="cuda", generator=g, dtype=dtype)
    out, shape = kernels.ttm(S, [P, D, Q], 1, U)
    ref = torch.einsum("pdq,nd->pnq", S.double(), U.double())
    mag = torch.einsum("pdq,nd->pnq", S.double().abs(), U.double().abs())
    assert shape == [P, n, Q]
    assert torch.all((out.double() - ref).abs() <= 2 * (D + 1) * eps * mag + 1e-30)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("P,D,Q,n", F32)
def test_f32(P, D, Q, n, shift):
    check(P, D, Q, n, torch.float32, 2.0 ** -24, shift)


F64 = [(3, 5, 15, 18), (1, 14, 15, 40), (1, 31, 33, 70), (1, 32, 33, 70), (200, 14, 24, 1), (60, 14, 8, 8),
       (200, 40, 8, 33), (200, 40, 8, 32), (200, 40, 15, 48), (200, 40, 15, 49), (1100, 33, 8, 64), (3, 300, 100, 100),
       (20, 300, 33, 64), (3000, 33, 1, 14), (300, 40, 12, 33), (300, 40, 13, 49), (300, 40, 33, 9), (60, 40, 100, 30),
       (60, 87, 127, 104), (5, 100, 1, 64), (1, 7, 1, 1), (1, 40, 9000, 9)]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("P,D,Q,n", F64)
def test_f64(P, D, Q, n, shift):
    check(P, D, Q, n, torch.float64, 2.0 ** -53, shift)
