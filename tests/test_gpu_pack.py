"""The packing kernel at the edges of its tiles (1024 entries in 1 to 32 columns):
row-major and column-major factors, ranks around powers of two, against
torch.cat of the transposes, bit for bit."""
import pytest
import torch

from tensorfox_gb300 import autograd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("R", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 65])
def test_pack(R, dtype):
    dims = [1, 1024, 1025, 31, 32, 33, 129, 2049, 63, 65, 255, 513]
    g = torch.Generator(device="cuda").manual_seed(R)
    W = [torch.randn((d, R), device="cuda", dtype=dtype, generator=g) for d in dims]
    W = [w if l % 2 else w.t().contiguous().t() for l, w in enumerate(W)]
    ref = torch.cat([w.t().reshape(-1) for w in W])
    assert torch.equal(autograd._flat(W), ref)
    assert torch.equal(autograd._flat(W[:2]), ref[:R * 1025])
