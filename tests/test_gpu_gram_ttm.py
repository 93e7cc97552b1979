"""The mode Gram (``kernels.mode_gram``) and the FP64 mode product
(``kernels.ttm``) at the edges of their tiles, against FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (P, D, Q): rows around 8 / 32 / 64 tiles, contraction lengths around the 32-step
# chunk, the last mode (Q = 1), 16-byte and one-element copies
VIEWS = [(1, 2, 3), (1, 8, 31), (1, 9, 32), (3, 32, 33), (2, 33, 65), (5, 63, 7), (1, 64, 200), (4, 65, 36),
         (1, 129, 1000), (40, 100, 1), (33, 31, 1), (1000, 130, 1), (7, 200, 20), (300, 40, 2)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("P,D,Q", VIEWS)
def test_mode_gram_edges(P, D, Q, dtype):
    from tensorfox_gb300 import kernels
    g = torch.Generator(device="cuda").manual_seed(P + 3 * D + 7 * Q)
    for shift in (0, 1):     # one element off the 16-byte boundary
        S = torch.randn(P * D * Q + shift, device="cuda", generator=g, dtype=dtype)[shift:].view(P, D, Q)
        M = S.double().movedim(1, 0).reshape(D, -1)
        ref, mag = M @ M.t(), M.abs() @ M.t().abs()
        G = kernels.mode_gram(S, [P, D, Q], 1).double()
        # one rounding a product and a term, FP32 chains capped by the split
        n, u = (min(P * Q, 4096) + 16, 2.0 ** -24) if dtype == torch.float32 else (2 * P * Q + 16, 2.0 ** -53)
        assert torch.all((G - ref).abs() <= n * u * mag + 1e-30), shift
        assert torch.equal(G, G.t())


@pytest.mark.parametrize("n", [1, 4, 9, 20, 33, 70])
@pytest.mark.parametrize("P,D,Q", [(1, 5, 8), (1, 40, 33), (3, 33, 9), (70, 20, 64), (1, 64, 9000), (50, 31, 1),
                                   (3000, 34, 1), (6, 10, 3)])
def test_ttm_f64_edges(P, D, Q, n):
    from tensorfox_gb300 import kernels
    g = torch.Generator(device="cuda").manual_seed(P + 3 * D + 7 * Q + n)
    for shift in (0, 1):
        S = torch.randn(P * D * Q + shift, device="cuda", generator=g, dtype=torch.float64)[shift:].view(P, D, Q)
        U = torch.randn((n, D), device="cuda", generator=g, dtype=torch.float64)
        out, shape = kernels.ttm(S, [P, D, Q], 1, U)
        ref = torch.einsum("pdq,nd->pnq", S, U)
        mag = torch.einsum("pdq,nd->pnq", S.abs(), U.abs())
        assert shape == [P, n, Q]
        assert torch.all((out - ref).abs() <= 2 * (D + 1) * 2.0 ** -53 * mag + 1e-300), shift
