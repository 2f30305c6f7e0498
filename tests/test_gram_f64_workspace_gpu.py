"""The workspace of the real FP64 pencil (gram_i8_f64.cu): a large context holds
nothing beside its bundles for it (the pencil is formed in the temporary), a
small one at most 192 MB (the matrices and the allocator's grain aside); and fewer bands than the context's give the same
bands as a context of that size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _held(qsb, N, n):
    import torch
    free0 = torch.cuda.mem_get_info()[0]
    es = qsb.EigenSolver(N, n, False, "fp64")
    held = free0 - torch.cuda.mem_get_info()[0]
    es.close()
    return held


@pytest.mark.parametrize("n,N,extra", [(128, 96 ** 3, 32 << 20), (64, 96 ** 3, 32 << 20), (40, 64 ** 3, 224 << 20),
                                       (40, 16 ** 3, 224 << 20)])
def test_memory_of_a_context(qsb, n, N, extra):
    import torch
    torch.cuda.empty_cache()
    _held(qsb, 64, 1)                                    # kernels loaded
    handles = _held(qsb, 64, 1)                          # what the library handles take
    assert _held(qsb, N, n) - handles <= 5 * 8 * n * N + extra


@pytest.mark.parametrize("grid", [(12, 12, 12), (40, 36, 30)])
def test_fewer_bands_than_the_context(qsb, grid):
    import torch
    nx, ny, nz = grid
    N, h, n = nx * ny * nz, 0.4, 40
    gen = torch.Generator(device="cuda").manual_seed(nx)
    H = qsb.Hamiltonian(nx, ny, nz, h, h, h)
    H.set_potential(torch.rand(N, dtype=torch.float64, device="cuda", generator=gen))
    X0 = torch.rand(n, N, dtype=torch.float64, device="cuda", generator=gen) - 0.5
    qsb.orthonormalize(X0, N, h ** 3)
    evs = []
    for nmax in (n, 90):
        es = qsb.EigenSolver(N, nmax, False, "fp64")
        es.set_hamiltonian(H)
        X, keep, ev = X0.clone(), torch.zeros_like(X0), np.zeros(n)
        es.lobpcg_d(h ** 3, n, 3, ev, X, keep, True)
        evs.append(np.sort(ev))
    assert np.abs(evs[0] - evs[1]).max() < 1e-10 * np.abs(evs[0]).max()
    assert qsb.device_status() == 0
