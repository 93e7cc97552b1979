"""The FP64 Gram with more tiles than a wave of the SMs (at least four splits,
fewer where the contraction has fewer chunks), against FP64."""
import pytest
import torch

from tensorfox_gb300 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,D,Q", [(1, 1300, 129), (130, 1297, 1), (31, 1500, 1), (33, 700, 2), (65, 1255, 1),
                                   (1, 640, 40), (200, 1000, 1)])
def test_gram_f64(P, D, Q):
    g = torch.Generator(device="cuda").manual_seed(P + 3 * D + 7 * Q)
    S = torch.randn((P, D, Q), device="cuda", generator=g, dtype=torch.float64)
    M = S.movedim(1, 0).reshape(D, -1)
    G = kernels.mode_gram(S, [P, D, Q], 1)
    assert torch.all((G - M @ M.t()).abs() <= (2 * P * Q + 16) * 2.0 ** -53 * (M.abs() @ M.t().abs()))
    assert torch.equal(G, G.t())
