"""The one-launch pencil solve of the FP64 solvers (pencil_small.cu) through
LOBPCG calls, at pencil sizes around its limits (one band; the largest sizes of one
CTA and the first ones past them, which take the library) and on spectra with
exact degeneracies (a constant potential: free electrons).

Bars: after 3 iterations the Ritz values equal those of an FP64 torch LOBPCG of the
same start to 1e-10 relative; bands come back dV-orthonormal to 1e-9 (the
overlap of the last basis, conditioned up to 1e6, times rounding); every step by
the Cholesky route."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pencil(U, AU, n):
    import torch
    A, S = U.conj() @ AU.T, U.conj() @ U.T
    d = 1.0 / torch.sqrt(torch.diagonal(S).real)
    A, S = 0.5 * (A + A.mH) * d[:, None] * d, 0.5 * (S + S.mH) * d[:, None] * d
    L = torch.linalg.cholesky(S)
    B = torch.linalg.solve_triangular(L, A, upper=False)
    B = torch.linalg.solve_triangular(L, B.mH, upper=False)
    w, v = torch.linalg.eigh(0.5 * (B + B.mH))
    return w[:n], (torch.linalg.solve_triangular(L.mH, v[:, :n], upper=True) * d[:, None]).T


def _ritz_values(apply, X, dV, iters, cplx):
    """Ritz values of `iters` LOBPCG steps (no kept directions), in torch."""
    import torch
    X = X * math.sqrt(dV)
    AX, P, AP = apply(X), None, None
    R = AX - (X.conj() * AX).sum(1, keepdim=True).real * X
    n = len(X)
    for _ in range(iters):
        AR = apply(R)
        U, AU = torch.cat([X, R] if P is None else [X, R, P]), torch.cat([AX, AR] if P is None else [AX, AR, AP])
        w, C = _pencil(U, AU, n)
        P, AP = C[:, n:] @ U[n:], C[:, n:] @ AU[n:]
        X, AX = C[:, :n] @ X + P, C[:, :n] @ AX + AP
        R = AX - w[:, None] * X
    return w


@pytest.mark.parametrize("cplx,n", [(False, 1), (False, 2), (False, 11), (False, 16), (False, 31), (False, 32),
                                    (False, 43), (True, 1), (True, 3), (True, 24), (True, 26), (True, 27)])
@pytest.mark.parametrize("flat", [False, True])
def test_ritz_values_and_orthonormal_bands(qsb, cplx, n, flat):
    import torch
    m, h = 16, 0.4
    N, dV = m ** 3, h ** 3
    g = (0.3, -0.2, 0.5) if cplx else (0.0, 0.0, 0.0)
    gen = torch.Generator(device="cuda").manual_seed(n)
    H = qsb.Hamiltonian(m, m, m, h, h, h)
    H.set_potential(torch.zeros(N, dtype=torch.float64, device="cuda") if flat else
                    torch.rand(N, dtype=torch.float64, device="cuda", generator=gen))
    X = torch.rand((n, 2, N) if cplx else (n, N), dtype=torch.float64, device="cuda", generator=gen) - 0.5
    qsb.orthonormalize(X, N, dV, cplx)

    def apply(Z):
        p = torch.stack((Z.real, Z.imag), 1).contiguous() if cplx else Z.contiguous()
        o = torch.empty_like(p)
        H.apply(p, o, cplx, g)
        return torch.complex(o[:, 0], o[:, 1]) if cplx else o

    X0 = torch.complex(X[:, 0], X[:, 1]) if cplx else X.clone()
    ref = _ritz_values(apply, X0, dV, 3, cplx).cpu().numpy()
    es = qsb.EigenSolver(N, n, cplx, "fp64")
    es.set_hamiltonian(H, g)
    keep, ev = torch.zeros_like(X), np.zeros(n)
    if cplx:
        es.lobpcg_z(dV, n, 3, ev, X, keep, 0, 0.0, 0)
    else:
        es.lobpcg_d(dV, n, 3, ev, X, keep, True)
    assert es.solve_stats() == (3, 0)
    Z = torch.complex(X[:, 0], X[:, 1]) if cplx else X
    G = (Z.conj() @ Z.T * dV).cpu().numpy()
    assert np.abs(G - np.eye(n)).max() < 1e-9
    assert np.allclose(np.sort(ev), ref, rtol=1e-10, atol=1e-10)


def _cell(qsb, n, V, h=0.4, m=16):
    import torch
    H = qsb.Hamiltonian(m, m, m, h, h, h)
    H.set_potential(V)
    es = qsb.EigenSolver(m ** 3, n, False, "fp64")
    es.set_hamiltonian(H)
    return H, es


def _bands(qsb, n, dV, m=16):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(1)
    V = torch.rand(m ** 3, dtype=torch.float64, device="cuda", generator=gen)
    X = torch.rand(n, m ** 3, dtype=torch.float64, device="cuda", generator=gen) - 0.5
    qsb.orthonormalize(X, m ** 3, dV)
    return V, X


def test_equal_bands_stay_defined(qsb):
    """Two equal bands make the overlap singular: whichever way its pivots round, the
    steps are solved and the bands stay finite."""
    import torch
    n, dV = 6, 0.4 ** 3
    V, X = _bands(qsb, n, dV)
    X[3] = X[2]
    H, es = _cell(qsb, n, V)
    ev = np.zeros(n)
    es.lobpcg_d(dV, n, 2, ev, X, torch.zeros_like(X), True)
    chol, basis = es.solve_stats()
    assert chol + basis == 2 and np.all(np.isfinite(ev)) and bool(torch.isfinite(X).all())


def test_indefinite_overlap_takes_the_overlap_basis(qsb):
    """Kept directions of zero make the overlap's last pivots zero, exactly: the step is
    solved on the rest of the basis, whose Ritz values numpy gives."""
    import torch
    n, dV = 6, 0.4 ** 3
    V, X = _bands(qsb, n, dV)
    H, es = _cell(qsb, n, V)
    apply = lambda Z: H.apply(Z.contiguous(), torch.empty_like(Z))
    AX = apply(X)
    R = AX - (X * AX).sum(1, keepdim=True) * dV * X
    U = torch.cat([X, R / torch.linalg.norm(R, dim=1, keepdim=True)])
    A, S = (U @ apply(U).T).cpu().numpy(), (U @ U.T).cpu().numpy()
    L = np.linalg.cholesky(S)
    T = np.linalg.solve(L, np.linalg.solve(L, 0.5 * (A + A.T)).T)
    ref = np.linalg.eigvalsh(0.5 * (T + T.T))[:n]
    ev = np.zeros(n)
    es.lobpcg_d(dV, n, 1, ev, X, torch.zeros_like(X), False)
    assert es.solve_stats() == (0, 1)
    assert np.abs(np.sort(ev) - ref).max() < 1e-10 * np.abs(ref).max()


@pytest.mark.parametrize("n", [2, 12])
def test_unresolved_vectors_take_the_library(qsb, n):
    """An operator of 2^-470 (lengths of 2^235): the inverse iteration's squares overflow,
    the one-launch solve reports vectors it cannot make orthonormal, and the library's
    solution of the same pencil comes back: the Ritz values of the unscaled operator."""
    import torch
    V, X0 = _bands(qsb, n, 1.0)
    out = []
    for s in (0, 235):
        H, es = _cell(qsb, n, V * 2.0 ** (-2 * s), h=2.0 ** s * 0.4)
        X, ev = X0.clone(), np.zeros(n)
        es.lobpcg_d(1.0, n, 1, ev, X, torch.zeros_like(X), True)
        assert es.solve_stats() == (1, 0)
        assert float((X @ X.T - torch.eye(n, dtype=torch.float64, device="cuda")).abs().max()) < 1e-10
        out.append(np.sort(ev) * 2.0 ** (2 * s))
    assert np.abs(out[0] - out[1]).max() < 1e-10 * np.abs(out[0]).max()
