"""The MTTKRP (``mttkrp``, GaussNewton.py:411-423) at the edges of its tiles and
plans, in FP32 and FP64, against the same product in FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows around 32 / 64 / 128 and the short modes' limit, inner extents around the
# 32-step chunk, ranks around the column blocks, 16- and 4-byte copies, an
# inner group with and without outer modes, orders 2 to 5
SHAPES = [((17, 5, 7), 1), ((33, 31, 32), 8), ((32, 33, 64), 9), ((128, 20, 36), 16), ((129, 18, 35), 17),
          ((64, 65, 19), 50), ((40, 96, 33), 64), ((24, 50, 31), 65), ((20, 21, 22), 129), ((300, 17), 5),
          ((18, 19, 20, 21), 7), ((17, 3, 18, 2, 19), 12), ((20, 700, 90), 24), ((30, 1, 40), 6)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dims,R", SHAPES)
def test_mttkrp_edges(dims, R, dtype):
    import tensorfox_gb300 as tfx
    g = torch.Generator(device="cuda").manual_seed(sum(dims) + R)
    L = len(dims)
    # an offset of one element: the tensor's base is not 16-byte aligned
    for shift in (0, 1):
        buf = torch.randn(int(np.prod(dims)) + shift, device="cuda", generator=g, dtype=dtype)
        T = buf[shift:].view(dims)
        W = [torch.randn((d, R), device="cuda", generator=g, dtype=dtype) for d in dims]
        s = "abcde"[:L]
        for l in range(L):
            rest = [m for m in range(L) if m != l]
            eq = s + "," + ",".join(s[m] + "r" for m in rest) + "->" + s[l] + "r"
            ref = torch.einsum(eq, T.double(), *[W[m].double() for m in rest])
            mag = torch.einsum(eq, T.double().abs(), *[W[m].double().abs() for m in rest])
            out = tfx.mttkrp(T, W, l).double()
            # sums of K products of L factors: at most (K + L) roundings of the
            # sum of magnitudes (FP32: K capped by the split's chain); the FP64
            # reference has as many
            K = int(np.prod([dims[m] for m in rest]))
            n, u = (min(K, 4096) + L + 64, 2.0 ** -24) if dtype == torch.float32 else (2 * (K + L), 2.0 ** -53)
            assert torch.all((out - ref).abs() <= n * u * mag + 1e-30), (l, shift)


# cuts after the first, a middle and the last mode, halves of one and of several
# modes, short modes (whose single product takes a group too)
ALL_SHAPES = [((200, 31, 33), 20), ((31, 33, 200), 20), ((70, 75, 80), 50), ((40, 41, 3, 3), 64), ((3, 40, 41), 9),
              ((21, 22, 23, 24), 12), ((9, 10, 11, 12, 13), 5), ((5, 6, 4, 5, 3, 4), 3), ((50, 60), 7), ((12, 2, 500), 66)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dims,R", ALL_SHAPES)
def test_mttkrp_all_modes(dims, R, dtype):
    import tensorfox_gb300 as tfx
    from tensorfox_gb300.autograd import mttkrp_all, _flat
    g = torch.Generator(device="cuda").manual_seed(sum(dims) + R)
    L = len(dims)
    T = torch.randn(dims, device="cuda", generator=g, dtype=dtype)
    W = [torch.randn((d, R), device="cuda", generator=g, dtype=dtype) for d in dims]
    # the flat layout from factors of any strides
    flat = torch.cat([w.t().reshape(-1) for w in W])
    assert torch.equal(_flat(W), flat)
    assert torch.equal(_flat([w.t().contiguous().t() for w in W]), flat)
    assert torch.equal(_flat([torch.stack([w, w], 2)[:, :, 1] for w in W]), flat)
    every = mttkrp_all(T, flat, list(dims), R)
    s = "abcdef"[:L]
    for l in range(L):
        rest = [m for m in range(L) if m != l]
        eq = s + "," + ",".join(s[m] + "r" for m in rest) + "->" + s[l] + "r"
        ref = torch.einsum(eq, T.double(), *[W[m].double() for m in rest])
        mag = torch.einsum(eq, T.double().abs(), *[W[m].double().abs() for m in rest])
        # the GEMM's chain, then the group's contraction: at most one rounding a
        # product and a term
        K = int(np.prod([dims[m] for m in rest]))
        n, u = (min(K, 4096) + 2 * L + 64, 2.0 ** -24) if dtype == torch.float32 else (2 * (K + 2 * L), 2.0 ** -53)
        for out in (every[l], tfx.mttkrp(T, W, l)):
            assert torch.all((out.double() - ref).abs() <= n * u * mag + 1e-30), l
