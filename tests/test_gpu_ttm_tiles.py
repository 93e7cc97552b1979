"""The tensor-core mode product at the edges of its 128- and 256-wide tiles, on
either side of the rule between them, with several tiles a CTA (both pairs of
accumulators reused) and chunk counts from one, against FP64."""
import pytest
import torch

from tensorfox_gb300 import _lib, kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,D,Q,n", [(1, 32, 128, 1), (1, 64, 132, 16), (2, 96, 252, 33), (3, 32, 256, 64),
                                     (3, 160, 260, 50), (2, 64, 384, 31), (1, 128, 388, 32), (1, 512, 1000, 50),
                                     (500, 32, 128, 5), (310, 64, 300, 40), (7, 32, 25604, 64),
                                     (160, 64, 132, 16), (100, 96, 252, 33), (60, 160, 260, 50), (152, 64, 128, 7),
                                     (153, 64, 128, 7), (1, 512, 19460, 64), (3, 64, 25604, 1)])
def test_product(P, D, Q, n):
    assert _lib.load().tfx_ttm_tc_supported(P, D, Q, n)
    g = torch.Generator(device="cuda").manual_seed(P + D + Q + n)
    T = torch.randn((P, D, Q), device="cuda", generator=g)
    U = torch.randn((n, D), device="cuda", generator=g)
    got, shape = kernels.ttm(T, [P, D, Q], 1, U, tensor_cores=True)
    kernels.check_ttm_flag()
    assert list(shape) == [P, n, Q]
    ref = torch.matmul(U.double(), T.double())
    mag = torch.matmul(U.double().abs(), T.double().abs())
    # a product loses lo * lo and the low parts' truncation (2^-20 + 2 * 2^-21);
    # each of the 3 D / 8 additions to the accumulator one truncation
    tol = 2.0 ** -19 + (3 * D / 8 + 8) * 2.0 ** -22
    assert float(((got.double().view(P, n, Q) - ref).abs() / mag).max()) <= tol
