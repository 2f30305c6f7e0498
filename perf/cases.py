"""Workloads of the Kohn-Sham H.psi / block LOBPCG / SCF path, through its public
entry points, at sizes from a 2-atom cell to a 54-atom supercell.

Each case is a dict of plain values.  prepare(case, seed) makes what a program
holds before the call (operator context, solver, bands on the device), run(state)
is one pass, work(case) the bytes and operations of a pass that no
implementation can leave out, exact(case, seed) the same outputs in 64-bit torch
without this package, tolerance(case) how far two correct implementations of
one precision differ.

Units: Hartree atomic units.  Pseudopotential of every bcc cell: analytic GTH
form, Z_ion 6, one s channel (r 0.4, h 5.0) and one p channel (r 0.55, h 1.5),
projector spheres of 6 r_l.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qumasun-workshop-template_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

A_BCC = 6.0
GTH = dict(nl=2, r=(0.40, 0.55), h=(5.0, 1.5), zion=6.0, rloc=0.45, c1=-4.0, c2=0.6)
# water's pseudopotentials: O with one s channel, H local only
GTH_O = dict(nl=1, r=(0.222, 0.0), h=(18.27, 0.0))
GTH_H = dict(nl=0, r=(0.0, 0.0), h=(0.0, 0.0))
RCUT = 6.0
KBT = 0.01


def listed():
    return [
        # H psi of the smallest production cell: 2-atom bcc, 32^3, 16 bands (one call of a
        # solver that is bound by launches and latency)
        dict(name="hpsi_bcc2_f64", op="hpsi", nx=32, ny=32, nz=32, h=0.1875, nb=16, atoms=2, dtype="f64", cplx=False,
             fft=False),
        # H psi at production size: 16-atom bcc supercell, 96^3, 128 real bands, FP64
        dict(name="hpsi_bcc16_f64", op="hpsi", nx=96, ny=96, nz=96, h=0.125, nb=128, atoms=16, dtype="f64", cplx=False,
             fft=False),
        # the mixed solver's operator on the 54-atom cell: 144^3, 384 bands, FP32
        dict(name="hpsi_bcc54_f32", op="hpsi", nx=144, ny=144, nz=144, h=0.125, nb=384, atoms=54, dtype="f32",
             cplx=False, fft=False),
        # one k-point of a 4 x 4 x 4 mesh: 48^3, 24 complex bands at a Bloch vector, FP32
        # (the mixed k-point solver's operator; the FP64 one runs inside lobpcg_kpt_f64)
        dict(name="hpsi_kpt_f32", op="hpsi", nx=48, ny=48, nz=48, h=0.125, nb=24, atoms=2, dtype="f32", cplx=True,
             fft=False),
        # a slab-like cell on an odd, uneven grid with an odd number of bands
        dict(name="hpsi_ragged_f64", op="hpsi", nx=45, ny=50, nz=63, h=0.2, nb=13, atoms=3, dtype="f64", cplx=False,
             fft=False),
        # the same operator with the FFT kinetic term (the reference's default), 96^3 x 128
        dict(name="hpsi_fft_f64", op="hpsi", nx=96, ny=96, nz=96, h=0.125, nb=128, atoms=16, dtype="f64", cplx=False,
             fft=True),
        # many small uneven cells at once (edges 32 to 64, 8 to 64 bands, 1 to 4 atoms each)
        dict(name="batch_f64", op="batch", systems=12, h=0.25, dtype="f64"),
        # one solver call of an SCF step (4 iterations), the FP64 drop-in at production size
        dict(name="lobpcg_bcc16_f64", op="lobpcg", nx=96, ny=96, nz=96, h=0.125, nb=128, atoms=16, prec="fp64",
             cplx=False, iters=4),
        # the same call in mixed precision (FP32 bundles, tensor-core Gram products and rotations)
        dict(name="lobpcg_bcc16_mixed", op="lobpcg", nx=96, ny=96, nz=96, h=0.125, nb=128, atoms=16, prec="mixed",
             cplx=False, iters=4),
        # one solver call at one k-point (48^3, 24 complex bands), FP64
        dict(name="lobpcg_kpt_f64", op="lobpcg", nx=48, ny=48, nz=48, h=0.125, nb=24, atoms=2, prec="fp64", cplx=True,
             iters=4),
        # three whole SCF steps of the 2-atom cell (solver, density, Hartree, LDA, occupations, mixing)
        dict(name="scf_bcc2_f64", op="scf", nx=32, ny=32, nz=32, h=0.1875, nb=16, atoms=2, prec="fp64", steps=3),
        # nonlocal energy and forces at the end of an SCF: 16-atom cell, 128 bands, FP64
        dict(name="forces_bcc16_f64", op="forces", nx=96, ny=96, nz=96, h=0.125, nb=128, atoms=16, dtype="f64",
             cplx=False),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    if rng.random() < 0.5:      # a cubic cell, edges as programs choose them
        n = rng.choice([v for v in (16, 24, 32, 36, 40, 48, 54, 56, 60, 64, 72, 80, 90, 96, 108, 112) if lo <= v <= hi])
        return n, n, n
    return tuple(_logint(rng, lo, hi) for _ in range(3))


def draw(rng):
    op = rng.choice(["hpsi"] * 6 + ["lobpcg"] * 3 + ["batch", "forces", "scf"])
    if op == "batch":
        return dict(op=op, systems=rng.randint(2, 12), h=rng.choice([0.2, 0.25]), dtype=rng.choice(["f64", "f32"]))
    if op == "hpsi":
        nx, ny, nz = _grid(rng, 16, 112)
        cplx = rng.random() < 0.4
        most = 96 ** 3 * 128 // (nx * ny * nz * (2 if cplx else 1))
        return dict(op=op, nx=nx, ny=ny, nz=nz, h=rng.choice([0.125, 0.1875, 0.2, 0.25]),
                    nb=_logint(rng, 1, max(1, min(160, most))), atoms=rng.randint(0, 8),
                    dtype=rng.choice(["f64", "f32"]), cplx=cplx, fft=rng.random() < 0.2)
    if op == "forces":
        nx, ny, nz = _grid(rng, 24, 96)
        cplx = rng.random() < 0.4
        return dict(op=op, nx=nx, ny=ny, nz=nz, h=rng.choice([0.125, 0.1875, 0.25]), nb=_logint(rng, 2, 96),
                    atoms=rng.randint(1, 8), dtype=rng.choice(["f64", "f32"]), cplx=cplx)
    nx, ny, nz = _grid(rng, 24, 64)
    if op == "scf":
        n = rng.choice([24, 32, 36, 40, 48])
        return dict(op=op, nx=n, ny=n, nz=n, h=rng.choice([0.1875, 0.2, 0.25]), nb=rng.randint(10, 24), atoms=2,
                    prec="fp64", steps=rng.randint(2, 3))
    cplx = rng.random() < 0.5
    return dict(op=op, nx=nx, ny=ny, nz=nz, h=rng.choice([0.125, 0.1875, 0.25]), nb=_logint(rng, 4, 48 if cplx else 96),
                atoms=rng.randint(1, 4), prec=rng.choice(["fp64", "mixed"]), cplx=cplx, iters=rng.randint(2, 4))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _cell(case):
    return tuple(case[k] * case["h"] for k in ("nx", "ny", "nz"))


def _positions(case, seed):
    """bcc supercells with thermal displacements N(0, 0.1 bohr); other cells at random."""
    rng = np.random.default_rng(seed + 17)
    L, na = _cell(case), case["atoms"]
    reps = round((na / 2) ** (1 / 3)) if na else 0
    if reps and 2 * reps ** 3 == na and all(abs(v - reps * A_BCC) < 1e-9 for v in L):
        pos = [np.array([i, j, k], float) * A_BCC + s for i in range(reps) for j in range(reps) for k in range(reps)
               for s in (0.0, 0.5 * A_BCC)]
        return np.array(pos) + rng.normal(0.0, 0.1, (na, 3))
    return rng.uniform(0.0, 1.0, (na, 3)) * np.array(L)


def _bloch(case):
    if not case.get("cplx"):
        return (0.0, 0.0, 0.0)
    return tuple(2 * math.pi / v * f for v, f in zip(_cell(case), (0.25, 0.5, 0.75)))   # a point of a 4 x 4 x 4 mesh


def _uniform(shape, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(shape, dtype=dtype, device="cuda", generator=g) - 0.5


def _dtype(case):
    return torch.float64 if case.get("dtype", "f64") == "f64" else torch.float32


def _potential(case, seed):
    return 2.0 * _uniform((case["nx"] * case["ny"] * case["nz"],), torch.float64, seed + 1000)


def _orthonormal(X, dV):
    """dV-orthonormal bands (Gram-Schmidt's, by Cholesky); X: [n, N] real or complex."""
    Lc = torch.linalg.cholesky((X @ X.mH) * dV)
    return torch.linalg.solve_triangular(Lc, X, upper=False).contiguous()


def _start(case, seed):
    """Starting states of a solver: seeded uniform bands, orthonormalised; [n, N] or [n, 2, N] planes."""
    N, nb = case["nx"] * case["ny"] * case["nz"], case["nb"]
    if not case.get("cplx"):
        return _orthonormal(_uniform((nb, N), torch.float64, seed), case["h"] ** 3)
    X = _uniform((nb, 2, N), torch.float64, seed)
    Z = _orthonormal(torch.complex(X[:, 0], X[:, 1]), case["h"] ** 3)
    return torch.stack((Z.real, Z.imag), dim=1).contiguous()


def _systems(case, seed):
    """The independent cells of a batch: each a case of its own (edges and band counts from the count alone)."""
    rng = random.Random(4 + case["systems"])
    return [dict(nx=n, ny=n, nz=n, h=case["h"], nb=nb, atoms=na, dtype=case["dtype"])
            for n, nb, na in ((rng.choice([32, 40, 48, 56, 64]), rng.randint(8, 64), rng.randint(1, 4))
                              for _ in range(case["systems"]))]


def _hamiltonian(case, seed):
    import qsb
    h = case["h"]
    H = qsb.Hamiltonian(case["nx"], case["ny"], case["nz"], h, h, h)
    H.set_potential(_potential(case, seed))
    if case["atoms"]:
        H.set_gth_projectors(_positions(case, seed), [0] * case["atoms"], [GTH["nl"]], [GTH["r"]], [GTH["h"]], RCUT)
    if case.get("fft"):
        H.set_kinetic(1)
    return H


def _occupations(case):
    """Fermi-like filling, two electrons in the lowest bands."""
    nb = case["nb"]
    return 2.0 / (np.exp((np.arange(nb) - 0.6 * nb) / max(1.0, 0.05 * nb)) + 1.0)


def prepare(case, seed):
    import qsb
    op = case["op"]
    if op == "batch":
        subs = _systems(case, seed)
        hams = [_hamiltonian(c, seed + 31 * i) for i, c in enumerate(subs)]
        psis = [_uniform((c["nb"], H.N), _dtype(c), seed + 31 * i) for i, (c, H) in enumerate(zip(subs, hams))]
        return dict(op=op, hams=hams, psis=psis, out=[torch.empty_like(p) for p in psis])
    N, nb, h = case["nx"] * case["ny"] * case["nz"], case["nb"], case["h"]
    planes = (nb, 2, N) if case.get("cplx") else (nb, N)
    if op in ("hpsi", "forces"):
        psi = _uniform(planes, _dtype(case), seed)
        return dict(op=op, H=_hamiltonian(case, seed), psi=psi, out=torch.empty_like(psi) if op == "hpsi" else None,
                    cplx=bool(case["cplx"]), g=_bloch(case), occ=_occupations(case), atoms=case["atoms"])
    X0 = _start(case, seed)
    state = dict(op=op, X0=X0, X=torch.empty_like(X0), keep=torch.zeros_like(X0), dV=h ** 3, nb=nb, N=N,
                 cplx=bool(case.get("cplx")), H=_hamiltonian(case, seed), occ=_occupations(case))
    state["es"] = qsb.EigenSolver(N, nb, state["cplx"], case["prec"])
    if op == "lobpcg":
        state["es"].set_hamiltonian(state["H"], _bloch(case))
        state["iters"] = case["iters"]
        return state
    state["steps"] = case["steps"]
    state["scf"] = scf = qsb.SCF(state["H"], state["es"], nb, 6.0 * case["atoms"])
    scf.set_gth_local(_positions(case, seed), [0] * case["atoms"], [GTH["zion"]], [GTH["rloc"]], [GTH["c1"]],
                      [GTH["c2"]])
    scf.set_smearing(KBT)
    return state


def _fixed(X, keep):
    """States and kept directions with each band's free sign (phase) fixed at the band's first grid point."""
    if X.dim() == 2:
        s = torch.sign(X[:, :1])
        return X * s, keep * s
    u = torch.complex(X[:, 0, :1], X[:, 1, :1]).conj()
    u = u / u.abs()
    return tuple(torch.stack((B[:, 0] * u.real - B[:, 1] * u.imag, B[:, 0] * u.imag + B[:, 1] * u.real), dim=1)
                 for B in (X, keep))


def run(s):
    import qsb
    if s["op"] == "hpsi":
        return s["H"].apply(s["psi"], s["out"], s["cplx"], s["g"])
    if s["op"] == "batch":
        return qsb.apply_batch(s["hams"], s["psis"], s["out"])
    if s["op"] == "forces":
        e, f = s["H"].nonlocal_energy_force(s["psi"], s["occ"], s["atoms"], s["cplx"], s["g"])
        return dict(energy=e, forces=f)
    s["X"].copy_(s["X0"])       # every pass is the first solver call from these states
    if s["op"] == "scf":
        e, ev, occ = s["scf"].run(s["X"], s["keep"], 4, s["steps"], 1e-14)
        return dict(energies=e, eigen_values=ev, occupations=occ, density=s["scf"].field(0))
    ev = np.zeros(s["nb"])
    if s["cplx"]:
        s["es"].lobpcg_z(s["dV"], s["nb"], s["iters"], ev, s["X"], s["keep"], 0, 0.0, 0)
        rho = qsb.density(s["X"], np.repeat(s["occ"], 2), s["N"])
    else:
        s["es"].lobpcg_d(s["dV"], s["nb"], s["iters"], ev, s["X"], s["keep"], True)
        rho = qsb.density(s["X"], s["occ"], s["N"])
    X, P = _fixed(s["X"], s["keep"])
    return dict(eigen_values=ev, states=X, directions=P, density=rho)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _sphere_points(case):
    return int(case["atoms"] * 4.0 / 3.0 * math.pi * (RCUT * GTH["r"][1] / case["h"]) ** 3)


def _hpsi_work(case, dtype=None):
    """psi read, H psi written, V and the projector tables read once; stencil (27 operations a point) or two FFTs,
    V psi, and two products with the 4 projectors of each atom."""
    N, c = case["nx"] * case["ny"] * case["nz"], 2 if case.get("cplx") else 1
    e = 4 if (dtype or case.get("dtype")) == "f32" else 8
    cols, pts = case["nb"] * c, _sphere_points(case)
    kinetic = 5.0 * math.log2(N) * 2 if case.get("fft") else 27.0
    return dict(bytes=float(2 * cols * N * e + N * e + pts * 4 * e), flops=float(cols) * (N * (kinetic + 2) + pts * 16.0))


def work(case):
    op = case["op"]
    if op == "batch":
        parts = [_hpsi_work(c) for c in _systems(case, 0)]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    if op == "hpsi":
        return _hpsi_work(case)
    N, c, nb = case["nx"] * case["ny"] * case["nz"], 2 if case.get("cplx") else 1, case["nb"]
    pts = _sphere_points(case)
    if op == "forces":
        e = 4 if case["dtype"] == "f32" else 8
        return dict(bytes=float(nb * c * min(N, pts) * e + pts * 16 * e), flops=float(nb * c) * pts * 4 * 8)
    its = case["iters"] if op == "lobpcg" else 4 * case["steps"]
    hp = _hpsi_work(case, "f32" if case["prec"] == "mixed" else "f64")
    # per iteration: H of the residuals, both pencils' upper halves, the four rotated bundles
    pencil = sum(2.0 * N * (m * nb * c) ** 2 for m in [2] + [3] * (its - 1))
    rotate = its * 12.0 * N * nb * nb * c * c
    bundles = 4 if op == "lobpcg" else 2     # states and kept directions in and out
    return dict(bytes=float(bundles * nb * c * N * 8 + N * 8 * (1 if op == "lobpcg" else 20)),
                flops=pencil + rotate + its * hp["flops"])


def tolerance(case):
    op = case["op"]
    if op in ("hpsi", "batch", "forces"):
        return dict(rel=4e-7, max=1e-5) if case["dtype"] == "f32" else dict(rel=1e-14, max=1e-12)
    if case["prec"] == "mixed":
        return dict(rel=1e-3, max=1e-2)
    return dict(rel=5e-11, max=5e-9)


# ---------------------------------------------------------------------------
# the same outputs in 64-bit torch
# ---------------------------------------------------------------------------
_W2 = (8064.0, -1008.0, 128.0, -9.0)     # eighth-order second difference, / 5040
_W1 = (672.0, -168.0, 32.0, -3.0)        # eighth-order first difference, / 840


class _Operator:
    """H = T + V + V_NL on [n, N] bands (complex at a Bloch vector)."""

    def __init__(self, case, seed, V=None):
        self.n = (case["nz"], case["ny"], case["nx"])
        self.h, self.g, self.fft = case["h"], _bloch(case), bool(case.get("fft"))
        self.V = _potential(case, seed) if V is None else V
        self.atoms = []
        for R in _positions(case, seed):
            self.atoms.append(self._projectors(R))

    def _projectors(self, R, grad=False):
        """(folded index, projectors [4, p] with the Bloch phase exp(i g.r), KB energies) of the atom at R."""
        rl, rmax, h = GTH["r"], RCUT * max(GTH["r"]), self.h
        ax = [torch.arange(math.floor((x - rmax) / h), math.ceil((x + rmax) / h) + 1, device="cuda") for x in R]
        Z, Y, X = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
        X, Y, Z = X.reshape(-1), Y.reshape(-1), Z.reshape(-1)
        v = torch.stack([(I.double() * h - float(x)) for I, x in zip((X, Y, Z), R)])
        r2 = (v * v).sum(0)
        m = r2 <= rmax * rmax
        X, Y, Z, v, r2 = X[m], Y[m], Z[m], v[:, m], r2[m]
        nz, ny, nx = self.n
        idx = X % nx + nx * (Y % ny + ny * (Z % nz))
        s = torch.exp(-r2 / (2 * rl[0] ** 2)) * (r2.sqrt() <= RCUT * rl[0]) * (
            math.sqrt(2.0) / (rl[0] ** 1.5 * math.sqrt(math.sqrt(math.pi) / 2)) / math.sqrt(4 * math.pi))
        p = torch.exp(-r2 / (2 * rl[1] ** 2)) * (r2.sqrt() <= RCUT * rl[1]) * (
            math.sqrt(2.0) / (rl[1] ** 2.5 * math.sqrt(3 * math.sqrt(math.pi) / 4)) * math.sqrt(3 / (4 * math.pi)))
        beta = torch.stack([s, p * v[0], p * v[1], p * v[2]])
        E = torch.tensor([GTH["h"][0]] + [GTH["h"][1]] * 3, dtype=torch.float64, device="cuda")
        if any(self.g):
            ph = self.h * (self.g[0] * X.double() + self.g[1] * Y.double() + self.g[2] * Z.double())
            phase = torch.polar(torch.ones_like(ph), ph)
        else:
            phase = None
        if not grad:
            return idx, beta if phase is None else beta * phase, E
        d = [torch.stack([-v[k] / rl[0] ** 2 * s] + [p * ((1.0 if k == w else 0.0) - v[w] * v[k] / rl[1] ** 2)
                                                     for w in range(3)]) for k in range(3)]
        return idx, [b if phase is None else b * phase for b in [beta] + d], E

    def _kinetic(self, psi):
        f = psi.reshape(-1, *self.n)
        h = self.h
        if self.fft:
            k2 = 0.0
            for ax, (n, g) in enumerate(zip(self.n, self.g[::-1])):
                m = torch.arange(n, device="cuda")
                G = 2 * math.pi / (n * h) * torch.where(2 * m > n, m - n, m).double() + g
                k2 = k2 + (G * G).reshape([-1 if a == ax else 1 for a in range(3)])
            t = torch.fft.ifftn(torch.fft.fftn(f.to(torch.complex128), dim=(1, 2, 3)) * (0.5 * k2), dim=(1, 2, 3))
            return (t if psi.is_complex() else t.real).reshape(psi.shape)
        g2 = sum(g * g for g in self.g)
        out = f * (-14350.0 / 5040.0 * 3 / (h * h) - g2)
        for ax in range(3):
            g = self.g[2 - ax]
            for m in range(1, 5):
                up, dn = torch.roll(f, -m, dims=ax + 1), torch.roll(f, m, dims=ax + 1)
                out += (up + dn) * (_W2[m - 1] / (5040.0 * h * h))
                if g:
                    out += (up - dn) * (2j * g * _W1[m - 1] / (840.0 * h))
        return (-0.5 * out).reshape(psi.shape)

    def __call__(self, psi, chunk=32):
        out = torch.empty_like(psi)
        for b in range(0, psi.shape[0], chunk):
            p = psi[b:b + chunk]
            o = self._kinetic(p) + self.V * p
            for idx, beta, E in self.atoms:
                c = (p[:, idx] @ beta.T) * (E * self.h ** 3)
                o.index_add_(1, idx, c @ beta.conj())
            out[b:b + chunk] = o
        return out


def _planes(Z):
    return torch.stack((Z.real, Z.imag), dim=1) if Z.is_complex() else Z


def _bands(psi, cplx):
    psi = psi.double()
    return torch.complex(psi[:, 0], psi[:, 1]) if cplx else psi


def _pencil(U, AU, n, scale):
    """Lowest n eigenpairs of (U^H A U, U^H U), coefficients as rows [n, m]."""
    A, S = (U.conj() @ AU.T) * scale, (U.conj() @ U.T) * scale
    A, S = 0.5 * (A + A.mH), 0.5 * (S + S.mH)
    d = 1.0 / torch.sqrt(torch.diagonal(S).real)     # unit diagonal first: same pairs, better conditioned
    A, S = A * d[:, None] * d, S * d[:, None] * d
    Lc = torch.linalg.cholesky(S)
    B = torch.linalg.solve_triangular(Lc, A, upper=False)
    B = torch.linalg.solve_triangular(Lc, B.mH, upper=False)
    w, v = torch.linalg.eigh(0.5 * (B + B.mH))
    C = torch.linalg.solve_triangular(Lc.mH, v[:, :n], upper=True) * d[:, None]
    return w[:n], C.T.contiguous()


def _lobpcg_real(H, X, P, dV, iters, first):
    def unit(B):
        return 1.0 / torch.sqrt((B * B).sum(1, keepdim=True) * dV)
    n = X.shape[0]
    X = X * unit(X)
    AX = H(X)
    AP = None if first else H(P)
    R = AX - (X * AX).sum(1, keepdim=True) * dV * X
    R = R * unit(R)
    for it in range(iters):
        AR = H(R)
        two = first and it == 0
        U, AU = torch.cat([X, R] if two else [X, R, P]), torch.cat([AX, AR] if two else [AX, AR, AP])
        _, C = _pencil(U, AU, n, dV)
        P, AP = C[:, n:] @ U[n:], C[:, n:] @ AU[n:]
        X, AX = C[:, :n] @ X + P, C[:, :n] @ AX + AP
        x, p = unit(X), unit(P)
        X, AX, P, AP = X * x, AX * x, P * p, AP * p
        eps = (X * AX).sum(1) * dV
        R = AX - eps[:, None] * X
    return eps, X, P


def _lobpcg_complex(H, X, dV, iters, mixed):
    n = X.shape[0]
    X = X * math.sqrt(dV)
    if mixed:
        X = X / torch.linalg.norm(X, dim=1, keepdim=True)
    AX = H(X)
    R = AX - (X.conj() * AX).sum(1, keepdim=True).real * X
    P = AP = None
    for it in range(iters):
        AR = H(R)
        U, AU = torch.cat([X, R] if P is None else [X, R, P]), torch.cat([AX, AR] if P is None else [AX, AR, AP])
        w, C = _pencil(U, AU, n, 1.0)
        P, AP = C[:, n:] @ U[n:], C[:, n:] @ AU[n:]
        X, AX = C[:, :n] @ X + P, C[:, :n] @ AX + AP
        R = AX - w[:, None] * X
    return w, X / (torch.linalg.norm(X, dim=1, keepdim=True) * math.sqrt(dV)), P


def _g2(case):
    k = [torch.fft.fftfreq(case[a], d=case["h"], device="cuda", dtype=torch.float64) * (2 * math.pi)
         for a in ("nz", "ny", "nx")]
    return k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2, k


def _local_potential(case, seed):
    """Fourier series of the GTH local parts, Nyquist planes of even grids left out."""
    G2, k = _g2(case)
    n = (case["nz"], case["ny"], case["nx"])
    r, z, c1, c2 = GTH["rloc"], GTH["zion"], GTH["c1"], GTH["c2"]
    e = torch.exp(-0.5 * G2 * r * r)
    v = torch.where(G2 > 0, -4 * math.pi * z * e / torch.where(G2 > 0, G2, torch.ones_like(G2)),
                    torch.full_like(G2, 2 * math.pi * z * r * r))
    v = v + (2 * math.pi) ** 1.5 * r ** 3 * e * (c1 + c2 * (3 - G2 * r * r))
    for ax, m in enumerate(n):
        if m % 2 == 0:
            v.index_fill_(ax, torch.tensor([m // 2], device="cuda"), 0.0)
    S = 0
    for X, Y, Z in _positions(case, seed):
        ph = k[0][:, None, None] * float(Z) + k[1][None, :, None] * float(Y) + k[2][None, None, :] * float(X)
        S = S + torch.polar(torch.ones_like(ph), -ph)
    return (torch.fft.ifftn(v * S).real / case["h"] ** 3).reshape(-1)


def _filter(case, f, factor):
    n = (case["nz"], case["ny"], case["nx"])
    return torch.fft.ifftn(torch.fft.fftn(f.reshape(n)) * factor).real.reshape(-1)


def _lda(rho):
    """Perdew-Zunger LDA, (rho eps_xc, v_xc), zero below 1e-8."""
    r = torch.clamp(rho, min=1e-8)
    rs = (3 / (4 * math.pi * r)) ** (1 / 3)
    ex = -0.75 * (9 / (4 * math.pi ** 2)) ** (1 / 3) / rs
    s = torch.sqrt(rs)
    hi = -0.1423 / (1 + 1.0529 * s + 0.3334 * rs)
    dhi = hi * hi * (1.0529 * 0.5 * s + 0.3334 * rs) / (3 * -0.1423)
    lr = torch.log(rs)
    lo = -0.0480 + 0.0311 * lr - 0.0116 * rs + 0.0020 * rs * lr
    dlo = -(0.0311 + (0.0020 - 0.0116) * rs + 0.0020 * rs * lr) / 3
    ec, dec = torch.where(rs >= 1, hi, lo), torch.where(rs >= 1, dhi, dlo)
    on = rho >= 1e-8
    zero = torch.zeros_like(rho)
    return torch.where(on, rho * (ex + ec), zero), torch.where(on, 4.0 / 3.0 * ex + ec + dec, zero)


def _fermi(eig, n_el):
    lo, hi = eig.min() - 1.0, eig.max() + 1.0
    for _ in range(200):
        mu = 0.5 * (lo + hi)
        occ = 2.0 / (np.exp(np.minimum((eig - mu) / KBT, 80.0)) + 1.0)
        lo, hi = (mu, hi) if occ.sum() < n_el else (lo, mu)
    return occ


def _scf(case, seed):
    dV, nb, n_el = case["h"] ** 3, case["nb"], 6.0 * case["atoms"]
    G2, _ = _g2(case)
    hart = torch.where(G2 > 0, 4 * math.pi / torch.where(G2 > 0, G2, torch.ones_like(G2)), torch.zeros_like(G2))
    kerk = 0.5 * G2 / (G2 + 0.8 ** 2)
    vloc = _local_potential(case, seed)
    X, P = _start(case, seed), None
    rho = (torch.tensor(np.clip(n_el - 2.0 * np.arange(nb), 0.0, 2.0), device="cuda")[:, None] * X * X).sum(0)
    H = _Operator(case, seed, V=vloc)
    energies, ins, res = [], [], []
    for step in range(case["steps"]):
        vhxc = _filter(case, rho, hart) + _lda(rho)[1]
        H.V = vloc + vhxc
        _, X, P = _lobpcg_real(H, X, P, dV, 4, step == 0)
        rq = ((X * H(X)).sum(1) / (X * X).sum(1)).cpu().numpy()
        occ = _fermi(rq, n_el)
        out = (torch.tensor(occ, device="cuda")[:, None] * X * X).sum(0)
        e = float(occ @ rq) + dV * float((0.5 * _filter(case, out, hart) * out + _lda(out)[0] - vhxc * out).sum())
        energies.append(e)
        ins.append(rho)
        res.append(out - rho)
        m = len(res)
        B = np.array([[float(a @ b) for b in res] for a in res])
        M = np.ones((m + 1, m + 1))
        M[:m, :m], M[m, m] = B / B.diagonal().max(), 0.0
        a = np.linalg.solve(M, np.eye(m + 1)[m])[:m]
        rho = sum(float(c) * v for c, v in zip(a, ins)) + _filter(case, sum(float(c) * v for c, v in zip(a, res)), kerk)
    return dict(energies=np.array(energies), eigen_values=rq, occupations=occ, density=out)


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        return [_Operator(c, seed + 31 * i)(_uniform((c["nb"], c["nx"] * c["ny"] * c["nz"]), _dtype(c),
                                                     seed + 31 * i).double())
                for i, c in enumerate(_systems(case, seed))]
    if op == "scf":
        return _scf(case, seed)
    N, nb, cplx = case["nx"] * case["ny"] * case["nz"], case["nb"], bool(case["cplx"])
    H = _Operator(case, seed)
    if op in ("hpsi", "forces"):
        psi = _uniform((nb, 2, N) if cplx else (nb, N), _dtype(case), seed)
    if op == "hpsi":
        return _planes(H(_bands(psi, cplx)))
    if op == "forces":
        Z, occ = _bands(psi, cplx), torch.tensor(_occupations(case), device="cuda")
        energy, forces = 0.0, np.zeros((case["atoms"], 3))
        for a, R in enumerate(_positions(case, seed)):
            idx, tables, E = H._projectors(R, grad=True)
            c = [(Z[:, idx] @ t.T) * case["h"] ** 3 for t in tables]
            energy += float((occ[:, None] * E * c[0].abs() ** 2).sum())
            for k in range(3):
                forces[a, k] = float((2 * occ[:, None] * E * (c[0].conj() * c[1 + k]).real).sum())
        return dict(energy=energy, forces=forces)
    X, dV = _bands(_start(case, seed), cplx), case["h"] ** 3
    if cplx:
        ev, X, P = _lobpcg_complex(H, X, dV, case["iters"], case["prec"] == "mixed")
    else:
        ev, X, P = _lobpcg_real(H, X, None, dV, case["iters"], True)
    rho = (torch.tensor(_occupations(case), device="cuda")[:, None] * X.abs() ** 2).sum(0)
    X, P = _fixed(_planes(X), _planes(P))
    return dict(eigen_values=ev, states=X, directions=P, density=rho)
