"""The FP64 form's tensor-core workspace under a small budget and on a device short of memory: the
engine takes a smaller one and its results stay the same bits."""
import ctypes
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from nonequilibriumgreensfunction_gb300 import Solver, capi, hamiltonian
from nonequilibriumgreensfunction_gb300.serving import Server

from conftest import REPO

pytestmark = pytest.mark.gpu


def _workspace(m, batch):
    """Bytes of the whole workspace (and a little): 252 M^2 a matrix, 2 batch of them up to 10^7 / M^2,
    and 72 M^2 for Gamma, of which there are at most batch."""
    cap = min(2 * batch, max(32, 10**7 // m**2))
    return m * m * (252 * cap + 72 * min(batch, cap))


# A budget that lacks an eighth, most and nearly all of the workspace.
@pytest.mark.parametrize("lacking", [0.12, 0.7, 0.9])
def test_served_results_do_not_depend_on_the_workspace(need_gpu, lacking):
    npx, n, batch = 4, 8, 8                                     # M = 256: workspace of 302 MB
    model = hamiltonian.wire_model(W=0.1, seed=3, flux=0.3, zeeman=0.01)
    es = np.linspace(-0.2, 0.25, 8)
    with Solver(npx, n, n, eta=1e-3, sr_tol=1e-10, max_batch=batch) as s:
        s.build_hamiltonian(model)
        want = s.solve_batch(es, 0.7, 0.2, 1e-3)
        v = ctypes.c_int64()
        assert s.lib.negf_estimate_device_bytes(ctypes.byref(s.params), ctypes.byref(v)) == capi.NEGF_OK
    budget = v.value + (64 << 20) - int(lacking * _workspace(4 * n * n, batch))
    with Server(precision="fp64", max_batch=batch, slots_per_geometry=1, eta=1e-3, hbm_budget_bytes=budget) as srv:
        rid = srv.submit_model(npx, n, n, model, es, 0.7, 0.2, 1e-3)
        srv.wait(rid, timeout=300)
        got = srv.result(rid)
        assert got["status"] == 0 and srv.stats()["bytes_used"] <= budget
    for k in ("T12", "EDensity", "HDensity", "Modec1", "Modec2", "DOSc1", "DOSc2"):
        assert np.array_equal(got[k], want[k]), k


_SHORT = """
import ctypes, json, sys
import numpy as np, torch
from nonequilibriumgreensfunction_gb300 import Solver, hamiltonian
npx, n, batch, workspace = 2, 10, 40, int(sys.argv[1])
model = hamiltonian.wire_model(W=0.1, seed=3, flux=0.3, zeeman=0.01)
def solver(k):
    s = Solver(npx, n, n, eta=1e-2, sr_tol=1e-6, max_batch=k)
    s.build_hamiltonian(model)
    return s
with solver(1) as s:          # the kernels are loaded
    s.solve_batch([0.1], 0.7, 0.2, 1e-3)
    v = ctypes.c_int64()
    s.params.max_batch = batch
    assert s.lib.negf_estimate_device_bytes(ctypes.byref(s.params), ctypes.byref(v)) == 0
hold = torch.empty(max(torch.cuda.mem_get_info()[0] - (v.value - int(0.6 * workspace)), 0), dtype=torch.uint8, device="cuda")
es = np.linspace(-0.3, 0.3, batch)
with solver(batch) as s:
    short = s.device_bytes() < v.value
    s.profile(True)
    r = s.solve_batch(es, 0.7, 0.2, 1e-3)
    tc = s.stats()["tc_launches"]
del hold
torch.cuda.empty_cache()
with solver(batch) as s:
    w = s.solve_batch(es, 0.7, 0.2, 1e-3)
    whole = s.device_bytes() == v.value
print(json.dumps(dict(short=short, whole=whole, tc=tc, same=all(bool(np.array_equal(r[k], w[k])) for k in w))))
"""


# All but the engine's own blocks and 0.4 of its workspace held by somebody else (in a process of its
# own, so that no other test's blocks are at hand).
def test_engine_on_a_device_short_of_memory(need_gpu):
    out = subprocess.run([sys.executable, "-c", _SHORT, str(_workspace(400, 40))], cwd=REPO, capture_output=True, text=True,
                         timeout=300, env=dict(os.environ, PYTHONPATH=REPO))
    assert out.returncode == 0, out.stderr[-2000:]
    got = json.loads(out.stdout.splitlines()[-1])
    assert got["short"] and got["whole"] and got["tc"] > 0 and got["same"], got
