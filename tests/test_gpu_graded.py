"""Wires whose sites hardly couple (half a cross-section behind a wall of high potential), in the
FP64 form: densities that are many orders of magnitude below their neighbours' keep their digits."""
import numpy as np
import pytest

from nonequilibriumgreensfunction_gb300 import Solver, hamiltonian
from oracle import negf_oracle as O

pytestmark = pytest.mark.gpu
ETA, F1, F2, DE = 1e-3, 0.7, 0.2, 1e-3


def _wire(npx, npy, npz, wall, ends, bias=0.0, bdg=False):
    """The upper half of the cross-section at `wall` eV: inside the wire, or in the end slices too (and
    so in the leads)."""
    v = np.zeros((npx, npy, npz))
    v[slice(None) if ends else slice(1, -1), :, npz // 2:] = wall
    v += np.linspace(bias, -bias, npx)[:, None, None]
    h, x = hamiltonian.build_from_model(npx, npy, npz, hamiltonian.wire_model(zeeman=0.01, flux=0.4, V=v))
    return hamiltonian.bdg(h, x, npy, npz) if bdg else (h, x)


# Tolerance: the FP64 form's 1e-9, of every site's own density (the oracle itself is within 3e-12 of an 80-bit result).
# With walls in the leads their self-energies are graded too, whether one decimation gives both leads
# or (with a bias) each has its own.
@pytest.mark.parametrize("npx,npy,npz,ends,bias", [(10, 4, 4, False, 0.0), (4, 4, 4, True, 0.0), (4, 4, 4, True, 0.02)])
def test_every_site_keeps_its_digits(need_gpu, npx, npy, npz, ends, bias):
    h, x = _wire(npx, npy, npz, 1e3, ends, bias)
    energy = 0.11
    with Solver(npx, npy, npz, eta=ETA, sr_tol=1e-10) as s:
        s.set_hamiltonian(h, x)
        rho = s.new_site_array(1)
        got = s.solve_batch([energy], F1, F2, DE, rho_n=rho)
        again = s.stats()["fallbacks"]
    opt = O.SolveOptions(eta=ETA, sr_tol=1e-10)
    cse = O.contact_self_energy(h, x, energy, opt)
    inv = np.stack([(energy + 1j * ETA) * np.eye(a.shape[0]) - a for a in h])
    inv[0] -= cse["SigmaL"]
    inv[-1] -= cse["SigmaR"]
    g = O.get_retarded_greens(inv, x)
    gnp = O.calculate_gnp(g["GRLef"], g["GRRgt"], cse["GammaL"], cse["GammaR"], F1, F2, with_offdiag=False)
    want = O.site_density(gnp["Gnd"], npy, npz) * DE / (2 * np.pi)
    assert got["status"][0] == 0 and again > 0
    assert want.max() > 1e9 * want.min()
    assert (np.abs(rho[..., 0] - want) <= 1e-9 * np.abs(want)).all()
    for lead in (0, 1):
        assert abs(got["DOSc%d" % (lead + 1)][0] - cse["dosc"][lead]) <= 1e-9 * abs(cse["dosc"][lead])


# Graded and plain wires in one batch, in runs and single: everything is what each has on its own.
@pytest.mark.parametrize("npx,npy,npz,more", [(6, 4, 4, {}), (6, 4, 4, dict(calc_spin=True, calc_currents=True)),
                                              (6, 3, 3, dict(calc_currents=True)), (6, 3, 4, dict(contact_type=3, norb=8))])
@pytest.mark.parametrize("ends", [False, True])
def test_graded_and_plain_wires_in_one_batch(need_gpu, npx, npy, npz, more, ends):
    bdg = "contact_type" in more
    wires = [_wire(npx, npy, npz, 1e5, ends, bdg=bdg), _wire(npx, npy, npz, 0.0, ends, bdg=bdg)]
    slots = np.array([0, 1, 1, 0, 0, 1, 0])
    energies = 0.05 + 0.02 * np.arange(len(slots))

    def solve(pick, batch):
        with Solver(npx, npy, npz, eta=ETA, sr_tol=1e-10, n_hamiltonians=2, max_batch=batch, **more) as s:
            for k, (h, x) in enumerate(wires):
                s.set_hamiltonian(h, x, slot=k)
            arrays = {"rho_n": s.new_site_array(2), "rho_p": s.new_site_array(2)}
            if "calc_currents" in more:
                arrays["currents"] = [s.new_site_array(2) for _ in range(3)]
            out = s.solve_batch(energies[pick], F1, F2, DE, slots=slots[pick], **arrays)
            out.update(fallbacks=s.stats()["fallbacks"])
            return out, arrays

    every, sites = solve(np.arange(len(slots)), len(slots))
    assert every.pop("fallbacks") > 0
    for slot in (0, 1):
        pick = np.flatnonzero(slots == slot)
        one, alone = solve(pick, len(pick))
        assert (one.pop("fallbacks") > 0) == (slot == 0)
        for k, v in one.items():
            assert np.array_equal(every[k][pick], v), (slot, k)
        for k, v in alone.items():
            assert np.array_equal(np.asarray(sites[k])[..., slot], np.asarray(v)[..., slot]), (slot, k)


def test_graded_wire_energy_by_energy(need_gpu):
    """The per-energy calls, with the columns of G kept, against the batch."""
    npx, n = 8, 4
    h, x = _wire(npx, n, n, 1e3, True)
    with Solver(npx, n, n, eta=ETA, sr_tol=1e-10, keep_g_columns=True) as s:
        s.set_hamiltonian(h, x)
        rho = s.new_site_array()
        r = s.energy_sweep(0.11, F1, F2, DE, rho)
        left, _ = s.g_columns()
        batch = s.new_site_array(1)
        b = s.solve_batch([0.11], F1, F2, DE, rho_n=batch)
    assert r["T12"] == b["T12"][0] and np.array_equal(rho, batch[..., 0])
    opt = O.SolveOptions(eta=ETA, sr_tol=1e-10)
    cse = O.contact_self_energy(h, x, 0.11, opt)
    inv = np.stack([(0.11 + 1j * ETA) * np.eye(a.shape[0]) - a for a in h])
    inv[0] -= cse["SigmaL"]
    inv[-1] -= cse["SigmaR"]
    want = O.get_retarded_greens(inv, x)["GRLef"]
    # per site: rows of the column block
    size = lambda a: np.linalg.norm(np.asarray(a).reshape(npx * n * n, 4 * 4 * n * n), axis=1)  # noqa: E731
    got = np.asarray(left).reshape(np.asarray(want).shape)
    assert (size(got - want) <= 1e-9 * size(want)).all()
