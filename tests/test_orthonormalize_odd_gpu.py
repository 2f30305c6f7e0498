"""qsb_orthonormalize on odd numbers of complex bands (the interleaved copy behind
an odd-sized workspace has to stay 16-byte aligned)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 9])
def test_odd_complex_bundles(qsb, n):
    import torch
    N, dV = 1000, 0.03
    X = torch.rand(n, 2, N, dtype=torch.float64, device="cuda") - 0.5
    qsb.orthonormalize(X, N, dV, True)
    Z = torch.complex(X[:, 0], X[:, 1])
    assert float((Z.conj() @ Z.T * dV - torch.eye(n, device="cuda")).abs().max()) < 1e-13
