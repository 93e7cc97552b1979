"""Derivatives through the gradient of ``cp_fit_loss`` with respect to the
gradient that comes in (forward-mode products by double backward, gradients of a
scaled loss), against the directional derivative and the loss's own gradient."""
import pytest
import torch

import tensorfox_gb300 as tfx

pytestmark = pytest.mark.gpu


def case(dtype, dims=(14, 9, 7), R=5):
    g = torch.Generator(device="cpu").manual_seed(sum(dims) + R)
    T = torch.randn(*dims, generator=g, dtype=torch.float64).to("cuda", dtype)
    W = [torch.randn(d, R, generator=g, dtype=torch.float64).to("cuda", dtype) for d in dims]
    V = [torch.randn(d, R, generator=g, dtype=torch.float64).to("cuda", dtype) for d in dims]
    return T, W, V


@pytest.mark.parametrize("dtype,eps", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
def test_jvp_is_the_directional_derivative(dtype, eps):
    T, W, V = case(dtype)
    out, jvp = torch.autograd.functional.jvp(lambda *w: tfx.cp_fit_loss(T, list(w)), tuple(W), tuple(V))
    leaves = [w.clone().requires_grad_(True) for w in W]
    loss = tfx.cp_fit_loss(T, leaves)
    grads = torch.autograd.grad(loss, leaves)
    terms = torch.cat([(g.double() * v.double()).reshape(-1) for g, v in zip(grads, V)])
    assert float(out) == float(loss.detach())
    # the same gradients: only the sums over their n entries are rounded differently
    assert abs(float(jvp) - float(terms.sum())) <= (terms.numel() + 4) * eps * float(terms.abs().sum())
    assert float(jvp) != 0.0


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_gradients_of_a_scaled_loss(dtype):
    T, W, _ = case(dtype, (6, 5, 4, 3), 4)
    W = [w.requires_grad_(l != 2) for l, w in enumerate(W)]
    wanted = [w for w in W if w.requires_grad]
    plain = torch.autograd.grad(tfx.cp_fit_loss(T, W), wanted)
    a = torch.tensor(2.0, dtype=dtype, device="cuda", requires_grad=True)
    grads = torch.autograd.grad(a * tfx.cp_fit_loss(T, W), wanted, create_graph=True)
    for g, p in zip(grads, plain):
        assert g.requires_grad
        assert torch.equal(g.detach(), 2 * p)  # a power of two: exact
        # d/da of a * grad is grad, entry by entry
        for e in ((0, 0), (-1, -1)):
            da, = torch.autograd.grad(g[e], a, retain_graph=True)
            assert float(da) == float(p[e])
