"""The projection and expansion kernels (per-thread sums, tensor-core form,
pipelined expansion) at the edges of their batches: point counts around 32, 256
and the 8192-point chunk, widths around 4, 8 and 16, band counts around the
column groups, points outside the cell, several entries of one atom on a grid
point.  Against dense FP64 products (1e-13 relative: sums of at most 1e4 terms);
FP32 bundles to 1e-6 (one FP32 rounding of each result)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRID = (30, 24, 20)


def _tables(rng, npts, widths):
    nx, ny, nz = GRID
    coords, beta, dbeta, energy = [], [], [], []
    for n, w in zip(npts, widths):
        c = np.stack([rng.integers(-nx, 2 * nx, n), rng.integers(-5, ny + 5, n), rng.integers(-3, nz, n)], 1)
        coords.append(c.astype(np.int32))
        beta.append(rng.uniform(-1, 1, (w, n)))
        dbeta.append(rng.uniform(-1, 1, (3, w, n)))
        energy.append(rng.uniform(0.5, 2, w))
    return coords, beta, dbeta, energy


def _dense(coords, beta, psi, h, g):
    """<beta|psi> dV per atom and the phased gather index."""
    nx, ny, nz = GRID
    out = []
    for c, b in zip(coords, beta):
        idx = c[:, 0] % nx + nx * (c[:, 1] % ny + ny * (c[:, 2] % nz))
        ph = np.exp(1j * h * (c @ np.asarray(g))) if psi.dtype.kind == "c" else np.ones(len(idx))
        out.append((idx, ph, (psi[:, idx] * ph) @ np.swapaxes(b, -1, -2) * h ** 3))
    return out


@pytest.mark.parametrize("npts,widths", [((1, 31, 32, 33), (4, 4, 4, 4)), ((255, 256, 257), (1, 4, 3)),
                                         ((8191, 8193, 0), (4, 2, 4)), ((700, 40), (5, 9)), ((300, 8200), (16, 12)),
                                         ((64,), (1,))])
@pytest.mark.parametrize("nb", [1, 5, 17, 40])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_nonlocal_apply_and_forces(qsb, npts, widths, nb, cplx, dtype):
    import torch
    rng = np.random.default_rng(nb + sum(npts))
    nx, ny, nz = GRID
    N, h, g = nx * ny * nz, 0.3, (0.4, -0.3, 0.2)
    coords, beta, dbeta, energy = _tables(rng, npts, widths)
    H = qsb.Hamiltonian(nx, ny, nz, h, h, h)
    cat = lambda L: np.concatenate([np.ascontiguousarray(a).ravel() for a in L])
    H.set_projectors(npts, widths, cat(coords), cat(beta), cat(energy))
    H.set_projector_gradients(cat(dbeta))
    dt = torch.float64 if dtype == "f64" else torch.float32
    p = torch.from_numpy(rng.uniform(-0.5, 0.5, (nb, 2, N) if cplx else (nb, N))).to("cuda", dt)
    ph = p.double().cpu().numpy()
    psi = ph[:, 0] + 1j * ph[:, 1] if cplx else ph
    tol = 1e-13 if dtype == "f64" else 1e-6
    if dtype == "f32":      # the tables are rounded to FP32 too
        beta = [b.astype(np.float32).astype(np.float64) for b in beta]
        dbeta = [b.astype(np.float32).astype(np.float64) for b in dbeta]
    kw = dict(is_complex=cplx, g=g if cplx else (0.0, 0.0, 0.0))
    ref = np.zeros_like(psi)
    for (idx, phase, c), b, e in zip(_dense(coords, beta, psi, h, g), beta, energy):
        np.add.at(ref.T, idx, ((c * e) @ b * phase.conj()).T)
    got = torch.zeros_like(p)
    H.nonlocal_apply(p, got, **kw)
    a = got.double().cpu().numpy()
    a = a[:, 0] + 1j * a[:, 1] if cplx else a
    assert np.linalg.norm(a - ref) <= tol * np.linalg.norm(ref)
    occ = rng.uniform(0, 2, nb)
    E, F = H.nonlocal_energy_force(p, occ, len(npts), **kw)
    c0 = [c for _, _, c in _dense(coords, beta, psi, h, g)]
    e_ref = sum(float(np.sum(occ[:, None] * e * np.abs(c) ** 2)) for c, e in zip(c0, energy))
    f_ref = np.zeros((len(npts), 3))
    for d in range(3):
        for k, (_, _, gd) in enumerate(_dense(coords, [b[d] for b in dbeta], psi, h, g)):
            f_ref[k, d] = np.sum(2 * occ[:, None] * energy[k] * (c0[k].conj() * gd).real)
    scale = max(1.0, float(np.abs(f_ref).max()))
    assert abs(E - e_ref) <= 1e-12 * abs(e_ref)
    assert np.abs(F - f_ref).max() <= 1e-12 * scale


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_infinite_bands_stay_in_their_spheres(qsb, dtype):
    """A band with an infinity spoils the points of the spheres that hold it and
    nothing else: neither other bands nor points outside those spheres."""
    import torch
    rng = np.random.default_rng(3)
    nx, ny, nz = GRID
    N = nx * ny * nz
    c0 = np.stack([np.arange(200) % nx, np.full(200, 3), np.arange(200) // nx], 1)
    c1 = np.stack([np.arange(200) % nx, np.full(200, 4), np.arange(200) // nx], 1)
    H = qsb.Hamiltonian(nx, ny, nz, 0.3, 0.3, 0.3)
    H.set_projectors([200, 200], [4, 4], np.concatenate([c0.ravel(), c1.ravel()]).astype(np.int32),
                     rng.uniform(0.5, 1, 1600), np.ones(8))
    dt = torch.float64 if dtype == "f64" else torch.float32
    p = torch.rand(9, N, dtype=dt, device="cuda")
    idx = lambda c: c[:, 0] + nx * (c[:, 1] + ny * c[:, 2])
    p[4, idx(c0)[50]] = float("inf")
    out = torch.zeros_like(p)
    H.nonlocal_apply(p, out)
    bad = ~torch.isfinite(out).cpu().numpy()
    expect = np.zeros((9, N), bool)
    expect[4, idx(c0)] = True
    assert np.array_equal(bad, expect)
