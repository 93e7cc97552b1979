"""``tfx_mttkrp`` with less scratch than its plan asks for (one partial and up) and
with scratch off the 16-byte boundary: the general kernel serves those, and less
than one partial is an error; against FP64."""
import ctypes

import pytest
import torch

from tensorfox_gb300 import _lib, autograd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,eps", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
@pytest.mark.parametrize("dims,R", [((70, 30, 40), 20), ((5, 300, 9), 65), ((20, 1, 33), 7), ((3, 4, 5, 6), 3)])
def test_general_kernel(dims, R, dtype, eps):
    lib = autograd._declare()
    g = torch.Generator(device="cuda").manual_seed(sum(dims) + R)
    T = torch.randn(dims, device="cuda", dtype=dtype, generator=g)
    W = [torch.randn((d, R), device="cuda", dtype=dtype, generator=g) for d in dims]
    flat, es, s = autograd._flat(W), T.element_size(), "abcd"[:len(dims)]
    dt, cd = (_lib.F64 if es == 8 else _lib.F32), (ctypes.c_int * len(dims))(*dims)
    for m, d in enumerate(dims):
        o = [i for i in range(len(dims)) if i != m]
        eq = s + "," + ",".join(s[i] + "z" for i in o) + "->" + s[m] + "z"
        ref = torch.einsum(eq, T.double(), *[W[i].double() for i in o])
        mag = torch.einsum(eq, T.double().abs(), *[W[i].double().abs() for i in o])
        full = int(lib.tfx_mttkrp_scratch_bytes(dt, len(dims), cd, R, m))
        for nb, shift in ((d * R * es, 0), (3 * d * R * es, 0), (max(full, d * R * es), es)):
            scratch = torch.empty(nb + 16, dtype=torch.uint8, device="cuda")
            out = torch.empty((R, d), dtype=dtype, device="cuda")
            _lib.check(lib.tfx_mttkrp(dt, T.data_ptr(), len(dims), cd, R, flat.data_ptr(), m, out.data_ptr(),
                                      scratch.data_ptr() + shift, nb, autograd._st()))
            tol = (T.numel() // d + len(dims) + 4) * eps * mag
            assert torch.all((out.t().double() - ref).abs() <= tol), (m, nb, shift)
        if full > d * R * es:
            with pytest.raises(_lib.TfxError):
                _lib.check(lib.tfx_mttkrp(dt, T.data_ptr(), len(dims), cd, R, flat.data_ptr(), m, out.data_ptr(),
                                          scratch.data_ptr(), d * R * es - 1, autograd._st()))
