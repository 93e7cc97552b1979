"""FP64 symmetric eigensolver on matrices whose squared differences leave the
range of the rotations' short form (scales 1e-145 and 1e145), against the same
matrix at scale one."""
import pytest
import torch

from tensorfox_gb300 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 12])
@pytest.mark.parametrize("scale", [1e-145, 1.0, 1e145])
def test_scaled_matrix(n, scale):
    g = torch.Generator().manual_seed(n)
    B = torch.randn((n, n), generator=g, dtype=torch.float64)
    A = B @ B.T
    ev, V = kernels.sym_eig((A * scale).cuda())
    ev, V = ev.cpu() / scale, V.cpu()
    # at most ten sweeps of n - 1 rounds, six roundings a round and entry
    tol = 10 * n * 6 * 2.0 ** -53
    nrm = float(torch.linalg.matrix_norm(A, 2))
    assert float((V @ V.T - torch.eye(n, dtype=torch.float64)).abs().max()) <= tol
    assert float((V @ A @ V.T - torch.diag(ev)).abs().max()) <= 2 * tol * nrm
