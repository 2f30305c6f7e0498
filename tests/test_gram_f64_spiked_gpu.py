"""The real FP64 pencil (gram_i8_f64.cu) of bands with one dominant grid point,
whose tails lie far below the scale of the digits: an error of <u|u> there mixes
the spike with its tail.

Bands: a spike s of 0.87 each, on a uniform random tail t of norm 0.49; operator: 1 on
the spikes' points and 1.37 elsewhere, so the lowest n Ritz vectors of one step are
the spikes exactly.  Relative errors e_x, e_r of <x|x> and <r|r> leave
0.43 (e_x - e_r) / 0.37 of a band's tail in them: 1.4e-14 with the digit products up to
i + j = 7 only, which make <x|x> low by N 2^-65.6 and <r|r> by a quarter of that.
Otherwise it is the rounding of the step's few operations: 1e-15 to 3e-15 of either
sign (a library product's errors leave up to 4e-14)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_spikes_separate_from_their_tails(qsb):
    import torch
    n, N = 36, 96 ** 3
    gen = torch.Generator(device="cuda").manual_seed(5)
    T = torch.rand(n, N, dtype=torch.float64, device="cuda", generator=gen) - 0.5
    at = torch.arange(n, device="cuda") * 20011 + 777
    T[:, at] = 0.0
    T /= torch.linalg.norm(T, dim=1, keepdim=True)          # largest value ~ 2e-3
    X = 0.49 * T
    X[torch.arange(n, device="cuda"), at] = 0.87
    a = torch.full((N,), 1.37, dtype=torch.float64, device="cuda")
    a[at] = 1.0

    class Raw:                                               # a device array at an address
        def __init__(self, ptr, shape):
            self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False), version=3)

    def op(nb, x, ax, stream):
        view = [torch.as_tensor(Raw(p, (nb, N)), device="cuda") for p in (x, ax)]
        torch.mul(view[0], a, out=view[1])
        return 0

    es = qsb.EigenSolver(N, n, False, "fp64")
    es.set_operator(op)
    ev, keep = np.zeros(n), torch.zeros_like(X)
    es.lobpcg_d(1.0, n, 1, ev, X, keep, True)
    assert np.abs(ev - 1.0).max() < 1e-13
    # the Ritz vectors span the spikes, in any rotation Q: the share of each spike's own tail
    Q = X[:, at]
    own = (Q.T @ (X @ T.T)).diagonal()
    assert abs(float(own.mean())) < 2e-15 and float(own.abs().max()) < 8e-15
    assert qsb.device_status() == 0
