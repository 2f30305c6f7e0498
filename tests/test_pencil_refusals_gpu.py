"""Pencils that must not reach the library's dense solvers (they may never come
back from entries that are not finite): a search basis with vanishing columns is
solved on the rest, one with NaN is refused.  Sizes on both sides of the
one-CTA solve's limits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _start(qsb, n, cplx, m=12, h=0.4):
    import torch
    N = m ** 3
    gen = torch.Generator(device="cuda").manual_seed(n)
    H = qsb.Hamiltonian(m, m, m, h, h, h)
    H.set_potential(torch.rand(N, dtype=torch.float64, device="cuda", generator=gen))
    X = torch.rand((n, 2, N) if cplx else (n, N), dtype=torch.float64, device="cuda", generator=gen) - 0.5
    qsb.orthonormalize(X, N, h ** 3, cplx)
    return H, X, N, h ** 3


@pytest.mark.parametrize("cplx,n", [(False, 8), (False, 40), (True, 8), (True, 40)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_vanishing_directions_are_dropped(qsb, cplx, n, prec):
    """Zero kept directions in a call that is not the first: the same step as the first call's."""
    import torch
    H, X0, N, dV = _start(qsb, n, cplx)
    out = []
    for first in (True, False):
        es = qsb.EigenSolver(N, n, cplx, prec)
        es.set_hamiltonian(H)
        X, keep, ev = X0.clone(), torch.zeros_like(X0), np.zeros(n)
        if cplx:
            es.lobpcg_z(dV, n, 1, ev, X, keep, 0, 0.0, 0 if first else 1)
        else:
            es.lobpcg_d(dV, n, 1, ev, X, keep, first)
        out.append(np.sort(ev))
        if not first:
            assert es.solve_stats()[1] == 1
    assert np.abs(out[0] - out[1]).max() < (1e-10 if prec == "fp64" else 1e-4) * np.abs(out[0]).max()


@pytest.mark.parametrize("n", [8, 40])
@pytest.mark.parametrize("straight", [False, True])
def test_a_pencil_of_nan_is_refused(qsb, n, straight):
    """Bands without any residual cannot be normalised: NaN directions.  straight: the
    overlap basis without the Cholesky route in front of it (another Gram kind)."""
    import torch
    _, X, N, dV = _start(qsb, n, False)
    es = qsb.EigenSolver(N, n, False, "fp64")
    if straight:
        es.set_gram_kind("bf16x3")

    class Raw:
        def __init__(self, ptr, shape):
            self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False), version=3)

    def zero(nb, x, ax, stream):
        y = torch.as_tensor(Raw(ax, (nb, N)), device="cuda")
        torch.mul(torch.as_tensor(Raw(x, (nb, N)), device="cuda"), 0.0, out=y)
        return 0

    es.set_operator(zero)
    with pytest.raises(qsb.QsbError, match="non-finite"):
        es.lobpcg_d(dV, n, 1, np.zeros(n), X, torch.zeros_like(X), True)
