"""A solve right after an upload works on the new wire, also while other processes keep the GPU and
its copy engines busy (each process has its turns, and what one left unfinished waits for the next)."""
import os
import subprocess
import sys

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

# Each process uploads two wires in turn into one handle of each kind, and into new handles, and
# solves at once; a result that is not that wire's own (from its first, synchronised solve) is printed.
_LOOP = """
import sys, time
import numpy as np, torch
from nonequilibriumgreensfunction_gb300 import Solver, hamiltonian
seed, seconds = int(sys.argv[1]), float(sys.argv[2])
kinds = [dict(npx=3, npy=3, npz=2, contact_type=1), dict(npx=3, npy=3, npz=3), dict(npx=3, npy=2, npz=2, precision="mixed"),
         dict(npx=2, npy=4, npz=4, contact_type=1)]
def solve(s):
    return s.solve_batch([0.11, 0.2], 0.7, 0.2, 1e-3)
work = []
for k, kind in enumerate(kinds):
    size = [kind[a] for a in ("npx", "npy", "npz")]
    wires = [hamiltonian.ti_wire(*size, W=0.3, seed=10 * seed + 2 * k + i, zeeman=0.01) for i in (0, 1)]
    wires[1] = (wires[1][0] + 0.05 * np.eye(wires[1][0].shape[1]), wires[1][1])
    s = Solver(**kind, eta=1e-3, max_batch=2)
    want = []
    for h, x in wires:
        s.set_hamiltonian(h, x)
        torch.cuda.synchronize()
        want.append(solve(s))
    work.append((kind, wires, want, s))
end, n, bad = time.time() + seconds, 0, 0
while time.time() < end:
    for kind, wires, want, s in work:
        for (h, x), w in zip(wires, want):
            s.set_hamiltonian(h, x)
            r = solve(s)
            bad += any(not np.array_equal(r[k], w[k]) for k in w)
            n += 1
        with Solver(**kind, eta=1e-3, max_batch=2) as new:
            new.set_hamiltonian(*wires[n % 2])
            r = solve(new)
            bad += any(not np.array_equal(r[k], want[n % 2][k]) for k in r)
            n += 1
print(n, bad)
"""


def test_solve_right_after_an_upload(need_gpu):
    procs = [subprocess.Popen([sys.executable, "-c", _LOOP, str(i), "12"], cwd=REPO, stdout=subprocess.PIPE, stderr=subprocess.PIPE,
                              text=True, env=dict(os.environ, PYTHONPATH=REPO)) for i in range(4)]
    for p in procs:
        out, err = p.communicate(timeout=300)
        assert p.returncode == 0, err[-2000:]
        n, bad = map(int, out.split())
        assert n > 100 and bad == 0, (n, bad)
