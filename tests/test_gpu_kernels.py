"""Edges of the device kernels' size ranges, against the oracle."""
import numpy as np
import pytest

from nonequilibriumgreensfunction_gb300 import Solver, capi, hamiltonian, scf
from oracle import negf_oracle as O

pytestmark = pytest.mark.gpu


def _one_energy(npx, npy, npz, precision, energy=0.11, eta=1e-3):
    htotd, hopx = hamiltonian.ti_wire(npx, npy, npz, W=0.1, seed=3, flux=0.4, zeeman=0.01)
    with Solver(npx, npy, npz, eta=eta, sr_tol=1e-10, precision=precision) as s:
        s.set_hamiltonian(htotd, hopx)
        rho = s.new_site_array(1)
        got = s.solve_batch([energy], 0.7, 0.2, 1e-3, rho_n=rho)
    opt = O.SolveOptions(eta=eta, sr_tol=1e-10)
    cse = O.contact_self_energy(htotd, hopx, energy, opt)
    m = htotd.shape[1]
    inv = np.stack([(energy + 1j * eta) * np.eye(m) - h for h in htotd])
    inv[0] -= cse["SigmaL"]
    inv[-1] -= cse["SigmaR"]
    g = O.get_retarded_greens(inv, hopx)
    y = g["GRRgt"][0] @ cse["GammaR"] @ g["GRRgt"][0].conj().T
    t12 = np.real(np.trace(cse["GammaL"] @ y))
    gnp = O.calculate_gnp(g["GRLef"], g["GRRgt"], cse["GammaL"], cse["GammaR"], 0.7, 0.2, with_offdiag=False)
    want = O.site_density(gnp["Gnd"], npy, npz) * 1e-3 / (2 * np.pi)
    assert got["status"][0] == 0
    return got["T12"][0], t12, rho[..., 0], want


# The FP32 panel holds a row per thread: a partial last warp and a last panel of fewer than 32
# columns (M = 4, 36, 140), the switch from 512 to 640 threads (512, 520), its last size (640)
# and the shared-memory panel beyond it (644).  Tolerance: the mixed form's 1e-6.
@pytest.mark.parametrize("npy,npz", [(1, 1), (3, 3), (5, 7), (8, 16), (10, 13), (10, 16), (7, 23)])
def test_mixed_form_at_the_panel_kernels_sizes(need_gpu, npy, npz):
    t, want, rho, rho_want = _one_energy(3, npy, npz, "mixed")
    assert abs(t - want) <= 1e-6 * max(abs(want), 1e-3)
    assert np.abs(rho - rho_want).max() <= 1e-6 * np.abs(rho_want).max()


# The FP64 form takes its products and inverses on the tensor cores from M = 32 (28 and 32)
# with one set of accumulators up to K = 400 and two up to 800, and on the FP64 pipe beyond.
# Tolerance: the FP64 form's 1e-9.
@pytest.mark.parametrize("npy,npz", [(1, 7), (2, 4), (3, 3), (1, 33), (10, 10), (1, 101), (10, 20), (3, 67)])
def test_fp64_form_at_its_path_switches(need_gpu, npy, npz):
    t, want, rho, rho_want = _one_energy(3, npy, npz, "fp64")
    assert abs(t - want) <= 1e-9 * max(abs(want), 1e-3)
    assert np.abs(rho - rho_want).max() <= 1e-9 * np.abs(rho_want).max()


# What a double holds and the slices' common scale of a row does not: a wall of 1e8 eV on a
# site (the FP64 form's 1e-9), and a NaN or an infinity in one sample, which stays in that
# sample and leaves its neighbour's bits alone.
@pytest.mark.parametrize("value", [1e8, np.nan, np.inf])
def test_fp64_form_with_extreme_entries(need_gpu, value):
    npx, npy, npz = 4, 3, 3
    htotd, hopx = hamiltonian.ti_wire(npx, npy, npz, W=0.1, seed=3, flux=0.4, zeeman=0.01)
    bad = htotd.copy()
    bad[1, 5, 5] = value
    with Solver(npx, npy, npz, eta=1e-3, sr_tol=1e-10, n_hamiltonians=2, max_batch=2) as s:
        s.set_hamiltonian(htotd, hopx, slot=0)
        s.set_hamiltonian(bad, hopx, slot=1)
        alone = s.solve_batch([0.11], 0.7, 0.2, 1e-3)
        both = s.solve_batch([0.11, 0.11], 0.7, 0.2, 1e-3, slots=[0, 1])
    assert both["T12"][0] == alone["T12"][0] and both["Modec1"][0] == alone["Modec1"][0]
    if np.isfinite(value):
        opt = O.SolveOptions(eta=1e-3, sr_tol=1e-10, kT=0.025)
        want = O.energy_sweep(bad, hopx, 0.11, (0.005, -0.005), 1e-3, npy, npz, opt)
        assert abs(both["T12"][1] - want["T12"]) <= 1e-9 * abs(want["T12"])
    else:
        assert np.isnan(both["T12"][1])


# Up to 40 Poisson grids take a cluster of CTAs each, more take one CTA: the same bits and the
# same number of steps, below, at and above one element per thread (1024 sites).
@pytest.mark.parametrize("shape", [(5, 1, 1), (9, 3, 4), (16, 8, 8), (41, 5, 5), (30, 9, 8)])
def test_poisson_cluster_gives_the_same_bits(need_gpu, shape):
    rho = 1e-3 * np.random.default_rng(1).standard_normal(shape + (41,))
    one_cta, steps = scf.poisson_solve(rho, (0.02, -0.02, 0.1), 1.8)
    cluster, few = scf.poisson_solve(rho[..., :40], (0.02, -0.02, 0.1), 1.8)
    last, more = scf.poisson_solve(rho[..., 40:], (0.02, -0.02, 0.1), 1.8)
    assert np.array_equal(one_cta[..., :40], cluster) and np.array_equal(one_cta[..., 40:], last)
    assert max(few, more) == steps


# FP64 solves up to M = 38 run in one kernel per phase, with a cluster of 8, 4, 2 or 1 CTAs per
# problem by their number (1, 12, 40, 80 energies): one channel of each orbital count, sizes at
# the ends and at the cluster threshold (1, 2, 15, 16, 36, 38) and the first beyond (39).  The
# same bits in every batch, and the oracle's values to the FP64 form's 1e-9.
@pytest.mark.parametrize("channel,npy,npz", [(2, 1, 1), (4, 1, 1), (2, 5, 3), (0, 2, 2), (0, 3, 3), (3, 19, 1), (2, 13, 3)])
def test_small_cross_sections_in_every_cluster(need_gpu, channel, npy, npz):
    npx, norb, eta = 5, hamiltonian.CHANNEL_NORB[channel], 1e-3
    model = hamiltonian.channel_model(channel, W=0.2, seed=4)
    htotd, hopx = hamiltonian.build_from_model(npx, npy, npz, model)
    energies = np.linspace(0.31, 0.73, 80) + (2.0 if channel == 2 else 0.0)
    runs = []
    for n in (80, 40, 12, 1):
        with Solver(npx, npy, npz, norb=norb, eta=eta, sr_tol=1e-10, max_batch=n) as s:
            s.build_hamiltonian(model)
            rho = s.new_site_array(1)
            runs.append((s.solve_batch(energies[:n], 0.7, 0.2, 1e-3, rho_n=rho), rho))
    for n, (r, _) in zip((40, 12, 1), runs[1:]):
        for k in r:
            assert np.array_equal(r[k], runs[0][0][k][:n]), k
    r, rho = runs[3]
    opt = O.SolveOptions(eta=eta, sr_tol=1e-10, norb=norb)
    cse = O.contact_self_energy(htotd, hopx, energies[0], opt)
    inv = np.stack([(energies[0] + 1j * eta) * np.eye(h.shape[0]) - h for h in htotd])
    inv[0] -= cse["SigmaL"]
    inv[-1] -= cse["SigmaR"]
    g = O.get_retarded_greens(inv, hopx)
    gnp = O.calculate_gnp(g["GRLef"], g["GRRgt"], cse["GammaL"], cse["GammaR"], 0.7, 0.2, with_offdiag=False)
    want = O.site_density(gnp["Gnd"], npy, npz, norb) * 1e-3 / (2 * np.pi)
    t12 = np.real(np.trace(cse["GammaL"] @ g["GRRgt"][0] @ cse["GammaR"] @ g["GRRgt"][0].conj().T))
    assert r["status"][0] == 0 and r["sr_iters"][0] == cse["sr_iters"].max()
    assert abs(r["T12"][0] - t12) <= 1e-9 * max(abs(t12), 1e-3)
    assert abs(r["DOSc1"][0] - cse["dosc"][0]) <= 1e-9 * abs(cse["dosc"][0])
    assert np.abs(rho[..., 0] - want).max() <= 1e-9 * np.abs(want).max()


# The FP64 inverse has panels of eight columns up to n = 1024 (the last of 1, 7 or 8); beyond, and in
# the mixed form's redone inverses, a few matrices have their panels on clusters of eight CTAs.  Tolerance: 100 n eps of the product of the norms; a zero column gives its INFO.
@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 1024, 1025])
def test_fp64_inverse_at_its_panel_sizes(need_gpu, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))
    x, info = capi.zinv(a)
    assert info == 0
    for m, i in zip(a, x):
        bound = 100 * n * np.finfo(float).eps * np.linalg.norm(m, 2) * np.linalg.norm(i, 2)
        assert np.abs(m @ i - np.eye(n)).max() <= bound
    a[1, :, n - 1] = 0.0
    assert capi.zinv(a)[1] == n


# The A side is sliced eight rows a block, 64 k a warp, its rows staged in shared memory (up to
# k = 800).  Tolerance: 8 k eps of the product of moduli (NumPy's own rounding), and for the slice
# pairs left out 8 S 2^(-7 S) k of a row's and a column's largest; row scales spread over 2^40.
@pytest.mark.parametrize("slices", [3, 5, 7, 8])
@pytest.mark.parametrize("m,k", [(1, 1), (7, 16), (8, 63), (9, 65), (33, 257), (17, 800)])
def test_sliced_rows_at_their_block_sizes(need_gpu, m, k, slices):
    rng = np.random.default_rng(m * k)
    a = rng.standard_normal((2, m, k)) + 1j * rng.standard_normal((2, m, k))
    a *= np.ldexp(1.0, rng.integers(-20, 20, (2, m, 1)))
    b = rng.standard_normal((2, k, 11)) + 1j * rng.standard_normal((2, k, 11))
    got = capi.zgemm(a, b, slices=slices)
    bound = 8 * k * np.finfo(float).eps * (np.abs(a) @ np.abs(b)) + k * 8 * slices * 2.0**(-7 * slices) * (
        np.abs(a).max(2, keepdims=True) * np.abs(b).max(1, keepdims=True))
    assert (np.abs(got - a @ b) <= bound).all()


# The FP32 inverse factorises a panel beside the update before it: a CTA a matrix up to one an SM,
# the panels before the tiles with more (M >= 256), and on their own with more small ones; tiles of 48
# columns outside the two panels.  No result depends on the batch: 160 energies at once (up to 320
# lead blocks) and four at a time give the same bits.
@pytest.mark.parametrize("npy,npz", [(3, 3), (5, 13), (5, 20)])
def test_inverses_do_not_depend_on_the_batch(need_gpu, npy, npz):
    htotd, hopx = hamiltonian.ti_wire(3, npy, npz, W=0.1, seed=3, flux=0.4, zeeman=0.01)
    energies = np.linspace(-0.3, 0.3, 160)
    out = []
    for batch in (160, 4):
        with Solver(3, npy, npz, eta=1e-2, sr_tol=1e-6, max_batch=batch, precision="mixed") as s:
            s.set_hamiltonian(htotd, hopx)
            pick = [energies] if batch == 160 else [energies[:4], energies[78:82], energies[-4:]]
            res = [s.solve_batch(e, 0.7, 0.2, 1e-3) for e in pick]
        out.append({k: np.concatenate([np.atleast_1d(r[k]) for r in res]) for k in ("T12", "Modec1", "sr_iters")})
    some = np.r_[0:4, 78:82, 156:160]
    for k, v in out[0].items():
        assert np.array_equal(v[some], out[1][k]), k


# The FP64 form's tensor-core workspace holds at most max(32, 10^7 / M^2) matrices: larger batches go
# through it in pieces (M = 400: 62 matrices; M = 576: 32), which no result shows.
@pytest.mark.parametrize("npy,npz,n", [(10, 10, 64), (12, 12, 33)])
def test_fp64_batches_beyond_the_workspace_give_the_same_bits(need_gpu, npy, npz, n):
    model = hamiltonian.wire_model(W=0.1, seed=3, flux=0.4, zeeman=0.01)
    energies = np.linspace(-0.3, 0.3, n)
    pick = np.r_[0, n // 2, n - 1]
    out = []
    for e in (energies, energies[pick]):
        with Solver(2, npy, npz, eta=1e-2, sr_tol=1e-6, max_batch=len(e)) as s:
            s.build_hamiltonian(model)
            out.append(s.solve_batch(e, 0.7, 0.2, 1e-3))
    for k, v in out[1].items():
        assert np.array_equal(out[0][k][pick], v), k


# Grids of fewer than 400 sites take clusters up to 20 at a time, of fewer than 640 up to 32: the same
# bits and steps on both sides of the lines.
@pytest.mark.parametrize("shape,most", [((5, 1, 1), 20), ((21, 19, 1), 20), ((20, 20, 1), 32), ((71, 9, 1), 32),
                                        ((16, 8, 5), 40)])
def test_poisson_small_grids_on_both_sides_of_the_lines(need_gpu, shape, most):
    rho = 1e-3 * np.random.default_rng(3).standard_normal(shape + (most + 1,))
    one_cta, steps = scf.poisson_solve(rho, (0.02, -0.02, 0.1), 1.8)
    cluster, few = scf.poisson_solve(rho[..., :most], (0.02, -0.02, 0.1), 1.8)
    last, more = scf.poisson_solve(rho[..., most:], (0.02, -0.02, 0.1), 1.8)
    assert np.array_equal(one_cta[..., :most], cluster) and np.array_equal(one_cta[..., most:], last)
    assert max(few, more) == steps
