"""How the tensor-core projection (nl_proj_mma_kernel) rounds its sums: a batch of
32 points is summed from zero and added to the running sum.

Every product is d / 4, d = 1 + 2^-45 - 2^-52, so a batch sums to 8 d exactly and
a running sum of such batches loses 2^-49 a step at most.  Running sums that took
every four points (d) would lose 2^-45 at each step past 256, 85 times per warp and
chunk of 8192 points: 7e-15 of the projection, 1.4e-14 of the energy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_running_sums_take_whole_batches(qsb):
    import torch
    n, atoms, npts, nb = 24, 40, 8192, 128          # 160 CTAs: the form for many columns
    d = 1.0 + 2.0 ** -45 - 2.0 ** -52
    rng = np.random.default_rng(1)
    H = qsb.Hamiltonian(n, n, n, 0.5, 0.5, 0.5)
    coords = rng.integers(0, n, (atoms * npts, 3)).astype(np.int32)
    H.set_projectors([npts] * atoms, [1] * atoms, coords.ravel(), np.full(atoms * npts, d / 4), np.ones(atoms))
    H.set_projector_gradients(np.zeros(3 * atoms * npts))
    psi = torch.ones(nb, n ** 3, dtype=torch.float64, device="cuda")
    occ = np.zeros(nb)
    occ[3] = 1.0
    e, f = H.nonlocal_energy_force(psi, occ, atoms)
    ref = atoms * (0.125 * npts * (d / 4)) ** 2      # a few roundings of 1e-16
    assert abs(e - ref) < 2e-15 * ref
    assert np.all(f == 0.0)
