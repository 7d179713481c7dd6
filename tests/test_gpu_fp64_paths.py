"""Which kernels the FP64 form takes by size and options, and what they do at the ends of their ranges:
entries that the slices' integers do not hold, decimations longer than one launch."""
import numpy as np
import pytest

from nonequilibriumgreensfunction_gb300 import Solver, capi, hamiltonian
from oracle import negf_oracle as O

pytestmark = pytest.mark.gpu


# One kernel per phase up to M = 38; from 39 on, or from 32 with currents, kept columns or
# superconducting contacts, sliced products on the tensor cores (in two accumulator sets beyond 400);
# the FP64 pipe below 32 and beyond 800.  Tolerance: the FP64 form's 1e-9.
@pytest.mark.parametrize("npy,npz,more,sliced", [(1, 7, dict(calc_currents=True), False), (2, 4, {}, False),
                                                 (2, 4, dict(calc_currents=True), True), (3, 3, {}, False),
                                                 (3, 3, dict(calc_currents=True), True), (3, 3, dict(keep_g_columns=True), True),
                                                 (2, 5, {}, True)])
def test_paths_by_size_and_options(need_gpu, npy, npz, more, sliced):
    npx, energy, eta, de = 4, 0.11, 1e-3, 1e-3
    h, x = hamiltonian.ti_wire(npx, npy, npz, W=0.1, seed=3, flux=0.4, zeeman=0.01)
    currents = "calc_currents" in more
    with Solver(npx, npy, npz, eta=eta, sr_tol=1e-10, **more) as s:
        s.set_hamiltonian(h, x)
        s.profile(True)
        rho = s.new_site_array(1)
        j = [s.new_site_array(1) for _ in range(3)] if currents else None
        got = s.solve_batch([energy], 0.7, 0.2, de, rho_n=rho, **(dict(currents=j) if currents else {}))
        assert (s.stats()["tc_launches"] > 0) == sliced
    opt = O.SolveOptions(eta=eta, sr_tol=1e-10)
    cse = O.contact_self_energy(h, x, energy, opt)
    inv = np.stack([(energy + 1j * eta) * np.eye(a.shape[0]) - a for a in h])
    inv[0] -= cse["SigmaL"]
    inv[-1] -= cse["SigmaR"]
    g = O.get_retarded_greens(inv, x)
    t12 = np.real(np.trace(cse["GammaL"] @ g["GRRgt"][0] @ cse["GammaR"] @ g["GRRgt"][0].conj().T))
    gnp = O.calculate_gnp(g["GRLef"], g["GRRgt"], cse["GammaL"], cse["GammaR"], 0.7, 0.2, with_offdiag=False)
    want = O.site_density(gnp["Gnd"], npy, npz) * de / (2 * np.pi)
    assert got["status"][0] == 0
    assert abs(got["T12"][0] - t12) <= 1e-9 * max(abs(t12), 1e-3)
    assert np.abs(rho[..., 0] - want).max() <= 1e-9 * np.abs(want).max()


# On the sliced path (M = 60, and 404 with two accumulator sets): a wall of 1e8 eV on an orbital (the
# FP64 form's 1e-9), and a NaN or an infinity in one sample, which stays in that sample and leaves its
# neighbour's bits alone.
@pytest.mark.parametrize("npy,npz", [(3, 5), (1, 101)])
@pytest.mark.parametrize("value", [1e8, np.nan, np.inf])
def test_sliced_path_with_extreme_entries(need_gpu, npy, npz, value):
    npx = 3
    h, x = hamiltonian.ti_wire(npx, npy, npz, W=0.1, seed=3, flux=0.4, zeeman=0.01)
    bad = h.copy()
    bad[1, 5, 5] = value
    with Solver(npx, npy, npz, eta=1e-3, sr_tol=1e-10, n_hamiltonians=2, max_batch=2) as s:
        s.set_hamiltonian(h, x, slot=0)
        s.set_hamiltonian(bad, x, slot=1)
        alone = s.solve_batch([0.11], 0.7, 0.2, 1e-3)
        s.profile(True)
        both = s.solve_batch([0.11, 0.11], 0.7, 0.2, 1e-3, slots=[0, 1])
        assert s.stats()["tc_launches"] > 0
    assert both["T12"][0] == alone["T12"][0] and both["Modec1"][0] == alone["Modec1"][0]
    if np.isfinite(value):
        opt = O.SolveOptions(eta=1e-3, sr_tol=1e-10, kT=0.025)
        want = O.energy_sweep(bad, x, 0.11, (0.005, -0.005), 1e-3, npy, npz, opt)
        assert abs(both["T12"][1] - want["T12"]) <= 1e-9 * abs(want["T12"])
    else:
        assert np.isnan(both["T12"][1])


# The same wire in other units, energies times 2^864 and 2^-864: whole rows beyond FP32 (whose inverses
# are redone) and, of the small ones, below what the strict exponents slice.  Transmission and modes do
# not depend on the unit; the densities scale with its inverse.  Tolerance: the FP64 form's 1e-9.
@pytest.mark.parametrize("power", [864, -864])
def test_sliced_path_in_other_units(need_gpu, power):
    npx, npy, npz, unit = 4, 3, 5, 2.0**power
    h, x = hamiltonian.ti_wire(npx, npy, npz, W=0.1, seed=3, flux=0.4, zeeman=0.01)
    out = []
    for u in (1.0, unit):
        with Solver(npx, npy, npz, eta=1e-3 * u, sr_tol=1e-10) as s:
            s.set_hamiltonian(h * u, x * u)
            s.profile(True)
            rho = s.new_site_array(1)
            r = s.solve_batch([0.11 * u], 0.7, 0.2, 1e-3, rho_n=rho)
            assert s.stats()["tc_launches"] > 0
            out.append((r, rho * u))
    (a, rho_a), (b, rho_b) = out
    assert b["status"][0] == 0 and b["sr_iters"][0] == a["sr_iters"][0]
    for k in ("T12", "Modec1", "Modec2"):
        assert abs(b[k][0] - a[k][0]) <= 1e-9 * abs(a[k][0]), k
    assert np.abs(rho_b - rho_a).max() <= 1e-9 * np.abs(rho_a).max()


# A lead at the edge of its band, without damping: H = 0, HopX = 1/2, E = 1 or -1.  Every decimation step
# leaves t = 1/2 and halves the change, in exact arithmetic, so a tolerance of 2^-200 takes 199 steps, in
# two launches of at most 128, and the self-energy is exactly E / 2.  A lead outside its band beside them
# (E = 3/2) is done early and stays as it is alone.  M = 1, 16 (a cluster of eight) and 38.
@pytest.mark.parametrize("npy,npz", [(1, 1), (4, 4), (19, 2)])
def test_decimations_longer_than_one_launch(need_gpu, npy, npz):
    npx, m = 3, npy * npz
    h = np.zeros((npx, m, m), complex)
    h[1] = 3.0 * np.eye(m)
    x = 0.5 * np.eye(m, dtype=complex)
    tol = 2.0**-200

    def solve(energies, cap):
        with Solver(npx, npy, npz, norb=1, eta=0.0, sr_tol=tol, sr_max_iter=cap, max_batch=len(energies)) as s:
            s.set_hamiltonian(h, x)
            return s.solve_batch(energies, 0.7, 0.2, 1e-3)

    outside = solve([1.5], 20000)
    assert outside["status"][0] == 0
    for cap in (127, 128, 129, 198, 199, 300):
        r = solve([1.0, 1.5, -1.0], cap)
        for i in (0, 2):
            assert r["sr_iters"][i] == min(cap, 199)
            assert r["status"][i] == (capi.NEGF_OK if cap >= 199 else capi.NEGF_ESR_NOCONV)
        for k, v in outside.items():
            assert r[k][1] == v[0], k
    with Solver(npx, npy, npz, norb=1, eta=0.0, sr_tol=tol) as s:
        s.set_hamiltonian(h, x)
        for energy in (1.0, -1.0):
            c = s.contact_self_energy(energy)
            for lead in ("SigmaL", "SigmaR"):
                assert np.array_equal(c[lead], 0.5 * energy * np.eye(m)), lead
