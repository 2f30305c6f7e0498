"""Bands whose squares overflow are refused by the real FP64 solver before any
pencil is formed: |x|^2 infinite (a band of 1e200), and |r|^2 infinite with a
finite Rayleigh quotient (a potential of 1e170).  The caller's bands come back
finite and the context goes on working."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 40])
@pytest.mark.parametrize("what", ["norm of x", "norm of r"])
def test_overflowing_norms_are_refused(qsb, n, what):
    import torch
    m, h = 8, 0.5
    N, dV = m ** 3, h ** 3
    gen = torch.Generator(device="cuda").manual_seed(n)
    V = torch.rand(N, dtype=torch.float64, device="cuda", generator=gen)
    X = torch.rand(n, N, dtype=torch.float64, device="cuda", generator=gen) - 0.5
    H = qsb.Hamiltonian(m, m, m, h, h, h)
    H.set_potential(V * 1e170 if what == "norm of r" else V)
    es = qsb.EigenSolver(N, n, False, "fp64")
    es.set_hamiltonian(H)
    bad = X.clone()
    if what == "norm of x":
        bad[n // 2] *= 1e200
    ev, keep = np.zeros(n), torch.zeros_like(X)
    with pytest.raises(qsb.QsbError, match="non-finite"):
        es.lobpcg_d(dV, n, 1, ev, bad, keep, True)
    assert bool(torch.isfinite(bad).all())
    H.set_potential(V)
    es.lobpcg_d(dV, n, 1, ev, X, keep, True)
    assert np.all(np.isfinite(ev)) and es.solve_stats()[0] == 1
