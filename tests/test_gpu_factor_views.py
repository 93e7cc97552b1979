"""Factors as a program may have them (transposed, strided, expanded, reversed
copies, views that torch negates lazily): the same results, bit for bit, as from
contiguous copies of their values."""
import pytest
import torch

import tensorfox_gb300 as tfx

pytestmark = pytest.mark.gpu


def views(dtype):
    g = torch.Generator(device="cpu").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64).to("cuda", dtype)  # noqa: E731
    z = torch.complex(rnd(9, 4), rnd(9, 4))
    return {"negated": z.conj().imag, "negated contiguous": torch._neg_view(rnd(9, 4)), "transposed": rnd(4, 9).t(),
            "strided": rnd(18, 8)[::2, 1::2], "expanded": rnd(9, 1).expand(9, 4)}


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("kind", ["negated", "negated contiguous", "transposed", "strided", "expanded"])
def test_same_as_a_copy(kind, dtype):
    A = views(dtype)[kind]
    assert A.is_neg() == kind.startswith("negated")
    copy = torch.empty((9, 4), dtype=dtype, device="cuda").copy_(A)
    rest = [torch.randn(d, 4, device="cuda", dtype=dtype) for d in (7, 5)]
    T = torch.randn(9, 7, 5, device="cuda", dtype=dtype)
    got, ref = [A] + rest, [copy] + rest
    assert torch.equal(tfx.cp_reconstruct(got), tfx.cp_reconstruct(ref))
    assert torch.equal(tfx.cp_fit_loss(T, got), tfx.cp_fit_loss(T, ref))
    for m in range(3):
        assert torch.equal(tfx.mttkrp(T, got, m), tfx.mttkrp(T, ref, m))
