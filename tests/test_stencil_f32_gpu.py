"""The TMA-fed FP32 stencil (fd8_wq_kernel) at the edges of its tiling: one tile,
tiles shifted back inside the grid, wrapped halos, few planes, z chunks, odd
band counts, grids it must leave to the register kernel.

Against the FP64 stencil of the same (FP32-valued) bands, itself pinned to the
reference: an FP32 sum of 26 terms whose magnitudes add up to S carries at most
~26 * 2^-24 S; S is below 4 |c0| max|psi|, and |L psi| is of the order
|c0| rms(psi), so 2e-6 of the result's root mean square in the L2 norm (observed
1e-7) and 2e-5 pointwise leave no room for a wrong neighbour (order 1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(32, 16, 4), (32, 32, 9), (48, 16, 8), (36, 20, 5), (64, 48, 33), (100, 36, 12), (144, 24, 17), (52, 84, 10),
         (28, 32, 8), (34, 32, 8), (40, 18, 6), (96, 96, 20)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("cplx", [False, True])
def test_f32_stencil_equals_f64(qsb, grid, cplx):
    import torch
    nx, ny, nz = grid
    N, nb, d, g = nx * ny * nz, 3, (0.2, 0.25, 0.21), (0.1, -0.2, 0.3)
    gen = torch.Generator(device="cuda").manual_seed(nx + 7 * ny + 31 * nz)
    shape = (nb, 2, N) if cplx else (nb, N)
    p = torch.rand(shape, dtype=torch.float32, device="cuda", generator=gen) - 0.5
    got = torch.full(shape, 0.5, dtype=torch.float32, device="cuda")
    ref = got.double()
    if cplx:
        qsb.laplacian_kpoint8th(got, p, -0.5, *d, g, grid)
        qsb.laplacian_kpoint8th(ref, p.double(), -0.5, *d, g, grid)
    else:
        qsb.laplacian8th(got, p, -0.5, *d, grid)
        qsb.laplacian8th(ref, p.double(), -0.5, *d, grid)
    V = torch.rand(N, dtype=torch.float64, device="cuda", generator=gen)
    H = qsb.Hamiltonian(nx, ny, nz, *d)
    H.set_potential(V.float().double())     # the same potential in both types
    hp, hp64 = torch.empty_like(p), torch.empty(shape, dtype=torch.float64, device="cuda")
    kw = dict(is_complex=cplx, g=g if cplx else (0.0, 0.0, 0.0))
    H.apply(p, hp, **kw)
    H.apply(p.double(), hp64, **kw)
    for a, b in ((got, ref), (hp, hp64)):
        e = (a.double() - b).cpu().numpy()
        rms = float(np.sqrt(np.mean(b.cpu().numpy() ** 2)))
        assert np.linalg.norm(e) / np.sqrt(e.size) < 2e-6 * rms
        assert np.max(np.abs(e)) < 2e-5 * rms
    assert qsb.device_status() == 0


# every form of both kernels: (complex, Bloch vector), += and V psi + forms, on grids with edge
# tiles, z chunks and odd band counts
SAME_BITS = r"""
import sys
import torch
import qsb
out = []
for nx, ny, nz, nb in [(32, 16, 4, 3), (48, 16, 8, 1), (36, 20, 5, 2), (64, 48, 33, 5), (100, 36, 12, 3), (52, 84, 40, 2),
                       (96, 96, 20, 7)]:
    N, d = nx * ny * nz, (0.2, 0.25, 0.21)
    gen = torch.Generator(device="cuda").manual_seed(nx + 7 * ny)
    V = torch.rand(N, dtype=torch.float64, device="cuda", generator=gen) - 0.5
    H = qsb.Hamiltonian(nx, ny, nz, *d)
    H.set_potential(V)
    for cplx, g in [(False, (0.0, 0.0, 0.0)), (True, (0.0, 0.0, 0.0)), (True, (0.1, -0.2, 0.3))]:
        p = torch.rand((nb, 2, N) if cplx else (nb, N), dtype=torch.float32, device="cuda", generator=gen) - 0.5
        a = torch.rand(p.shape, dtype=torch.float32, device="cuda", generator=gen)
        if cplx:
            qsb.laplacian_kpoint8th(a, p, -0.5, *d, g, (nx, ny, nz))
        else:
            qsb.laplacian8th(a, p, -0.5, *d, (nx, ny, nz))
        h = torch.empty_like(p)
        H.apply(p, h, is_complex=cplx, g=g)
        out += [a.cpu(), h.cpu()]
torch.save(out, sys.argv[1])
"""


def test_f32_stencil_equals_the_register_kernel_bit_for_bit(qsb, tmp_path):
    """fd8_wq_kernel against fd8_kernel (QSB_STENCIL=reg in a child process): the
    same FP32 contractions in the same order, whatever kernel a grid takes."""
    import os
    import subprocess
    import sys
    import torch
    pkg = os.path.dirname(os.path.abspath(qsb.__file__))
    res = []
    for variant in ("ws", "reg"):
        path = str(tmp_path / (variant + ".pt"))
        env = dict(os.environ, QSB_STENCIL=variant, PYTHONPATH=os.pathsep.join([pkg, os.environ.get("PYTHONPATH", "")]))
        r = subprocess.run([sys.executable, "-c", SAME_BITS, path], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        res.append(torch.load(path))
    assert len(res[0]) == len(res[1]) == 42
    for a, b in zip(*res):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
