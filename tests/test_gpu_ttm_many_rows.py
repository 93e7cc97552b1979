"""Mode products with more rows of U^T than a grid's third dimension counts tiles
of: an outer product (D = 1) is exact, so equality."""
import pytest
import torch

from tensorfox_gb300 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,Q,n", [(torch.float64, 1, 65535 * 32 + 1), (torch.float64, 8, 65535 * 32 + 1),
                                       (torch.float32, 129, 65535 * 64 + 1)])
def test_outer_product(dtype, Q, n):
    g = torch.Generator(device="cuda").manual_seed(Q)
    S = torch.randn((1, 1, Q), device="cuda", generator=g, dtype=dtype)
    U = torch.randn((n, 1), device="cuda", generator=g, dtype=dtype)
    out, shape = kernels.ttm(S, [1, 1, Q], 1, U)
    assert shape == [1, n, Q]
    assert torch.equal(out.view(n, Q), U * S.view(1, Q))
