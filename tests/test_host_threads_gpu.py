"""Two host threads, a context and a stream each, on problems whose kernels take
different amounts of shared memory from call to call (small pencils of both
kinds, FP32 stencil tiles, expansions over different numbers of atoms): no call
may fail, and every result equals the one of the thread running alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(qsb, n, cplx, grid, seed):
    import torch
    N, h = grid ** 3, 0.4
    gen = torch.Generator(device="cuda").manual_seed(seed)
    H = qsb.Hamiltonian(grid, grid, grid, h, h, h)
    H.set_potential(torch.rand(N, dtype=torch.float64, device="cuda", generator=gen))
    X0 = torch.rand((n, 2, N) if cplx else (n, N), dtype=torch.float64, device="cuda", generator=gen) - 0.5
    qsb.orthonormalize(X0, N, h ** 3, cplx)
    es = qsb.EigenSolver(N, n, cplx, "fp64")
    es.set_hamiltonian(H, (0.2, 0.1, -0.3) if cplx else (0.0, 0.0, 0.0))

    def run():
        X, keep, ev = X0.clone(), torch.zeros_like(X0), np.zeros(n)
        if cplx:
            es.lobpcg_z(h ** 3, n, 2, ev, X, keep, 0, 0.0, 0)
        else:
            es.lobpcg_d(h ** 3, n, 2, ev, X, keep, True)
        return X
    return run


def _apply(qsb, grid, nb, atoms, seed):
    import torch
    nx, ny, nz = grid
    N, h = nx * ny * nz, 0.3
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    H = qsb.Hamiltonian(nx, ny, nz, h, h, h)
    H.set_potential(torch.rand(N, dtype=torch.float64, device="cuda", generator=gen))
    H.set_gth_projectors(rng.uniform(0, 1, (atoms, 3)) * np.array(grid) * h, [0] * atoms, [2], [(0.4, 0.55)],
                         [(5.0, 1.5)], 6.0)
    p = torch.rand(nb, N, dtype=torch.float32, device="cuda", generator=gen) - 0.5

    def run():
        return H.apply(p, torch.empty_like(p))
    return run


@pytest.mark.parametrize("what", ["complex pencils", "real pencils", "applies"])
def test_no_call_disturbs_another_thread(qsb, what):
    import torch
    if what == "complex pencils":
        runs = [_solver(qsb, 16, True, 16, 1), _solver(qsb, 20, True, 16, 2)]
    elif what == "real pencils":
        runs = [_solver(qsb, 8, False, 16, 3), _solver(qsb, 21, False, 16, 4)]
    else:
        runs = [_apply(qsb, (32, 32, 16), 3, 1, 5), _apply(qsb, (48, 48, 16), 5, 6, 6)]
    alone = [r() for r in runs]
    torch.cuda.synchronize()
    errors, start = [], threading.Barrier(len(runs))

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for _ in range(40):
                    out = runs[k]()
                torch.cuda.current_stream().synchronize()
                if not torch.equal(out, alone[k]):
                    errors.append(f"thread {k}: another result")
        except Exception as e:      # noqa: BLE001 - reported by the assertion below
            errors.append(f"thread {k}: {e}")

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(runs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


FIRST = r"""
import threading
import torch
import qsb
n, nb, h = 32, 4, 0.3
N = n ** 3
psi = torch.rand(nb, N, dtype=torch.float64, device="cuda") - 0.5
V = torch.rand(N, dtype=torch.float64, device="cuda")
hams = []
for _ in range(8):
    H = qsb.Hamiltonian(n, n, n, h, h, h)
    H.set_potential(V)
    hams.append(H)
outs = [torch.empty_like(psi) for _ in hams]
torch.cuda.synchronize()
start = threading.Barrier(8)
def work(k):
    start.wait()
    hams[k].apply(psi, outs[k])
threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
[t.start() for t in threads]
[t.join() for t in threads]
torch.cuda.synchronize()
print(all(torch.equal(o, outs[0]) for o in outs))
"""


def test_first_calls_of_a_process_from_several_threads(qsb):
    """Every thread's first stencil finds the tensor-map encoder, whoever looked it up:
    without it a thread would take another kernel, with another rounding."""
    import os
    import subprocess
    import sys
    pkg = os.path.dirname(os.path.abspath(qsb.__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([pkg, os.environ.get("PYTHONPATH", "")]))
    for _ in range(3):
        r = subprocess.run([sys.executable, "-c", FIRST], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        assert r.stdout.strip().splitlines()[-1] == "True"
