"""Projector tables set again and again on one operator: memory comes back, and the
result is that of a fresh operator, from cells whose tables all share the small
allocation to ones with tables of several MB."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tables_are_replaced(qsb):
    import torch
    nx, ny, nz, h, nb = 48, 40, 36, 0.2, 3
    N = nx * ny * nz
    gen = torch.Generator(device="cuda").manual_seed(1)
    V = torch.rand(N, dtype=torch.float64, device="cuda", generator=gen)
    p = torch.rand(nb, N, dtype=torch.float64, device="cuda", generator=gen) - 0.5
    rng = np.random.default_rng(1)
    cell = np.array([nx, ny, nz]) * h
    sets = [(rng.uniform(0, 1, (na, 3)) * cell, r) for na, r in [(1, 0.05), (6, 0.55), (0, 0.3), (2, 0.3), (9, 0.6)]]

    def put(H, pos, r):
        H.set_gth_projectors(pos, [0] * len(pos), [2], [(0.8 * r, r)], [(5.0, 1.5)], 6.0)

    def apply(H):
        return H.apply(p, torch.empty_like(p))

    H = qsb.Hamiltonian(nx, ny, nz, h, h, h)
    H.set_potential(V)
    for pos, r in sets:                                   # the largest last: the workspace has its final size
        put(H, pos, r)
        got = apply(H)
        F = qsb.Hamiltonian(nx, ny, nz, h, h, h)
        F.set_potential(V)
        if len(pos):
            put(F, pos, r)
        assert torch.equal(got, apply(F))
        F.close() if hasattr(F, "close") else None
        del F
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(5):
        for pos, r in sets:
            put(H, pos, r)
            apply(H)
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= 8 << 20
