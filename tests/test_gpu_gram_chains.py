"""Accuracy of the FP32 Gram of the last mode over long contractions: rounding
errors no larger than those of chains of 1024 additions.  Against FP64, off the
diagonal (sums of independent terms): a chain of c additions is off by sqrt(c / 2)
roundings of 2^-24 / sqrt(3) in the mean square, relative to the terms' root sum of
squares."""
import pytest
import torch

from tensorfox_gb300 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,D", [(20000, 1000), (32768, 700), (65536, 700), (20000, 1500), (60000, 130), (262144, 512)])
def test_error_of_the_last_mode(K, D):
    g = torch.Generator(device="cuda").manual_seed(K + D)
    S = torch.randn((K, D, 1), device="cuda", generator=g)
    X = S.double().view(K, D)
    off = ~torch.eye(D, dtype=torch.bool, device="cuda")
    err = (kernels.mode_gram(S, [K, D, 1], 1).double() - X.t() @ X)[off]
    terms = ((X * X).t() @ (X * X))[off].sum().sqrt()
    assert float(err.norm() / terms) <= (1024 / 2) ** 0.5 * 2.0 ** -24 / 3 ** 0.5
