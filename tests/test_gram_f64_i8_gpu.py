"""The real FP64 pencil of 33 and more bands on the INT8 tensor cores
(gram_i8_f64.cu), through the steps of the real FP64 solver: band counts around its
128-column tiles, odd grids (columns off the 16-byte boundary), and a pencil whose
digits take two chunks of grid points.

One step from X, and one more from X and the kept P: the Ritz values against
numpy's of the same span (1e-11 relative to the largest: the entries agree to a few
1e-16 of |u||v|, times the conditioning of the overlap of random bands)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ritz(apply, bundles, n):
    import torch
    U = torch.cat([B / torch.linalg.norm(B, dim=1, keepdim=True) for B in bundles])
    A, S = (U @ apply(U).T).cpu().numpy(), (U @ U.T).cpu().numpy()
    L = np.linalg.cholesky(S)
    T = np.linalg.solve(L, np.linalg.solve(L, 0.5 * (A + A.T)).T)
    ref = np.linalg.eigvalsh(0.5 * (T + T.T))
    return ref[:n], np.abs(ref).max()


@pytest.mark.parametrize("n,grid", [(33, (8, 8, 8)), (33, (9, 9, 9)), (42, (21, 20, 13)), (43, (21, 20, 13)),
                                    (64, (25, 23, 21)), (65, (25, 23, 21)), (86, (25, 23, 21)), (128, (16, 16, 16)),
                                    (129, (27, 25, 23)), (171, (64, 64, 64))])
def test_ritz_values(qsb, n, grid):
    import torch
    nx, ny, nz = grid
    N, h = nx * ny * nz, 0.5
    dV = h ** 3
    gen = torch.Generator(device="cuda").manual_seed(n + nx)
    H = qsb.Hamiltonian(nx, ny, nz, h, h, h)
    H.set_potential(torch.rand(N, dtype=torch.float64, device="cuda", generator=gen))
    X = torch.rand(n, N, dtype=torch.float64, device="cuda", generator=gen) - 0.5
    # columns of very different extent: the digits' scale is a column's largest value
    X[::3] *= torch.exp(-40.0 * torch.rand(N, dtype=torch.float64, device="cuda", generator=gen))
    qsb.orthonormalize(X, N, dV)
    apply = lambda Z: H.apply(Z.contiguous(), torch.empty_like(Z))
    residual = lambda Z: apply(Z) - (Z * apply(Z)).sum(1, keepdim=True) * dV * Z
    es = qsb.EigenSolver(N, n, False, "fp64")
    es.set_hamiltonian(H)
    ev = np.zeros(n)
    keep = torch.zeros_like(X)

    ref, top = _ritz(apply, [X, residual(X)], n)
    es.lobpcg_d(dV, n, 1, ev, X, keep, True)
    assert np.abs(np.sort(ev) - ref).max() < 1e-11 * top

    if 3 * n < N // 2:
        ref, top = _ritz(apply, [X, residual(X), keep], n)
        es.lobpcg_d(dV, n, 1, ev, X, keep, False)
        assert np.abs(np.sort(ev) - ref).max() < 1e-11 * top
    assert qsb.device_status() == 0
