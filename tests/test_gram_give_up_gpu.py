"""A pencil whose tensor-core products gave up (a bounded wait that ran out) is
formed again by library products: the call returns the bands of that route, and
the device error word says what happened.  QSB_GRAM_F64_GIVE_UP in a child
process stands in for the wait: the host sets the words and a pencil of zeros
after the launches; nothing waits or fails on the GPU."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import json
import numpy as np
import torch
import qsb
m, n, h = 16, N_BANDS, 0.5
N, dV = m ** 3, h ** 3
gen = torch.Generator(device="cuda").manual_seed(3)
H = qsb.Hamiltonian(m, m, m, h, h, h)
H.set_potential(torch.rand(N, dtype=torch.float64, device="cuda", generator=gen))
X = torch.rand(n, N, dtype=torch.float64, device="cuda", generator=gen) - 0.5
qsb.orthonormalize(X, N, dV)
es = qsb.EigenSolver(N, n, False, "fp64")
es.set_hamiltonian(H)
ev, keep = np.zeros(n), torch.zeros_like(X)
es.lobpcg_d(dV, n, 3, ev, X, keep, True)
G = (X @ X.T * dV).cpu().numpy()
print(json.dumps(dict(ev=sorted(ev), stats=es.solve_stats(), word=qsb.device_status(clear=True),
                      orth=float(np.abs(G - np.eye(n)).max()))))
"""


def _run(n, **env):
    e = dict(os.environ, **env)
    e["PYTHONPATH"] = os.pathsep.join([os.path.join(ROOT, "qumasun-workshop-template_b200"), e.get("PYTHONPATH", "")])
    r = subprocess.run([sys.executable, "-c", CHILD.replace("N_BANDS", str(n))], env=e, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("n", [33, 50])      # first pencil solved in one CTA; library from the first on
def test_products_that_gave_up_are_formed_again(qsb, n):
    plain, forced = _run(n), _run(n, QSB_GRAM_F64_GIVE_UP="1")
    assert plain["word"] == 0 and forced["word"] == 2
    assert forced["stats"] == plain["stats"] == [3, 0]
    # two orders of sums of the same pencils, three steps
    assert max(abs(a - b) for a, b in zip(plain["ev"], forced["ev"])) < 1e-9
    assert forced["orth"] < 1e-9
