"""Handles used from several host threads at once: separate handles are independent, so each
thread's results are those it has alone, bit for bit."""
import threading

import numpy as np
import pytest

from nonequilibriumgreensfunction_gb300 import Solver, hamiltonian, scf

pytestmark = pytest.mark.gpu


def _together(works, calls):
    """Runs work() `calls` times in a thread of its own for each of `works`, all at once, and
    returns each thread's results (or what it raised)."""
    start = threading.Barrier(len(works))
    got = [[] for _ in works]

    def loop(work, out):
        start.wait()
        try:
            for _ in range(calls):
                out.append(work())
        except Exception as e:   # shown by the assertion of the caller
            out.append(e)
    threads = [threading.Thread(target=loop, args=a) for a in zip(works, got)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return got


def _same(got, alone):
    assert not isinstance(got, Exception), got
    for k, v in alone.items():
        assert np.array_equal(got[k], v), k


# A kernel's shared memory depends on the size of the wire: blocks of 400 and 576 orbitals
# (slices of A above 48 KB, both forms), 16 and 36 (the one-kernel phases, FP64), 40 and 144 (the
# fused FP32 inverse among them when the first call finds it faster).
@pytest.mark.parametrize("precision,sizes,calls", [("mixed", ((10, 10), (12, 12)), 25), ("fp64", ((10, 10), (12, 12)), 10),
                                                   ("fp64", ((2, 2), (3, 3)), 600), ("mixed", ((2, 5), (6, 6)), 60)])
def test_wires_of_two_sizes_at_once(need_gpu, precision, sizes, calls):
    solvers, works = [], []
    for npy, npz in sizes:
        model = hamiltonian.wire_model(W=0.1, seed=npy, flux=0.4, zeeman=0.01)
        s = Solver(2, npy, npz, eta=1e-2, sr_tol=1e-6, precision=precision)
        s.build_hamiltonian(model)
        solvers.append(s)
        works.append(lambda s=s: s.solve_batch([0.11], 0.7, 0.2, 1e-3))
    try:
        alone = [w() for w in works]
        for results, one in zip(_together(works, calls), alone):
            for r in results:
                _same(r, one)
            assert len(results) == calls
    finally:
        for s in solvers:
            s.close()


def test_poisson_grids_of_two_sizes_at_once(need_gpu):
    rng = np.random.default_rng(2)
    works = []
    for shape in ((9, 3, 4), (60, 12, 12)):
        rho = 1e-3 * rng.standard_normal(shape)
        works.append(lambda rho=rho: dict(zip(("U", "iters"), scf.poisson_solve(rho, (0.02, -0.02, 0.1), 1.8))))
    alone = [w() for w in works]
    for results, one in zip(_together(works, 400), alone):
        for r in results:
            _same(r, one)
        assert len(results) == 400
