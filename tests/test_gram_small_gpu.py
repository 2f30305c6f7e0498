"""The small real pencil formed in two launches (gram_small.cu), through the first
step of the real FP64 solver, at band counts around its tiles and limit (33 and
more bands take gram_i8_f64.cu) and grids around its 64-point chunks.

One iteration from dV-orthonormal bands: the Ritz values of span{X, R} against
numpy's (1e-11 relative to the largest: sums of at most 1e4 terms and the pencil's
conditioning)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 16, 21, 32, 33])
@pytest.mark.parametrize("grid", [(8, 8, 8), (9, 9, 9), (21, 20, 13)])
def test_first_ritz_values(qsb, n, grid):
    import torch
    nx, ny, nz = grid
    N, h = nx * ny * nz, 0.5
    dV = h ** 3
    gen = torch.Generator(device="cuda").manual_seed(n + nx)
    H = qsb.Hamiltonian(nx, ny, nz, h, h, h)
    H.set_potential(torch.rand(N, dtype=torch.float64, device="cuda", generator=gen))
    X = torch.rand(n, N, dtype=torch.float64, device="cuda", generator=gen) - 0.5
    qsb.orthonormalize(X, N, dV)
    apply = lambda Z: H.apply(Z.contiguous(), torch.empty_like(Z))
    AX = apply(X)
    R = AX - (X * AX).sum(1, keepdim=True) * dV * X
    U = torch.cat([X, R / torch.linalg.norm(R, dim=1, keepdim=True)])
    A, S = (U @ apply(U).T).cpu().numpy(), (U @ U.T).cpu().numpy()
    L = np.linalg.cholesky(S)
    T = np.linalg.solve(L, np.linalg.solve(L, 0.5 * (A + A.T)).T)
    ref = np.linalg.eigvalsh(0.5 * (T + T.T))
    es = qsb.EigenSolver(N, n, False, "fp64")
    es.set_hamiltonian(H)
    ev = np.zeros(n)
    es.lobpcg_d(dV, n, 1, ev, X, torch.zeros_like(X), True)
    assert np.abs(np.sort(ev) - ref[:n]).max() < 1e-11 * np.abs(ref).max()
