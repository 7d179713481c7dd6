"""The work that a user of this framework has it do, as cases to be timed and compared.

Three ways in, as the programs around the solver use them:

- ``sweep``: the reference's own energy loop, one ``Solver.energy_sweep`` per energy, with
  the site arrays accumulated on the host;
- ``batch``: the whole energy loop in one ``Solver.solve_batch``, in the FP64 form (the
  default) and in the mixed form, over several disorder samples (Hamiltonian slots);
- ``poisson``: the electrostatic step of the self-consistent loop, ``scf.poisson_solve``.

Geometries, materials, tolerances and energy windows are those of the repository's tests and
benchmark.  Every wire has its own Anderson disorder and energies, drawn from the seed.
"""
import math

import numpy as np
import torch

from nonequilibriumgreensfunction_gb300 import Solver, hamiltonian, scf

KT, MU1, MU2 = 0.025, 0.005, -0.005
# energy window of each channel model (eV): inside its bands
WINDOW = {"ti": (-0.2, 0.2), "ti_ref": (-0.4, 0.4), "surface": (0.1, 0.7), "soc": (-0.8, 0.8)}
NORB = {"ti": 4, "ti_ref": 4, "surface": 2, "soc": 2}


def _solve(name, kind, form, model, npx, npy, npz, energies, seeds=1, **more):
    # eta is 1e-5 eV in the mixed form.  In FP64 it is 1e-3: the decimation amplifies rounding as
    # eta falls, and at 1e-5 two FP64 solvers that are both right differ by 1e-7 and more near
    # the edge of a subband, so that there is nothing to compare.
    case = dict(name=name, kind=kind, form=form, model=model, npx=npx, npy=npy, npz=npz, energies=energies, seeds=seeds,
                eta=1e-5 if form == "mixed" else 1e-3, sr_tol=1e-10, W=0.1, spin=False, currents=False, bdg=False, bias=False)
    case.update(more)
    return case


def listed():
    return [
        # the smallest wire a user can ask for: the 1-D spin-orbit wire (M = 2), energy by energy
        _solve("sweep_soc_2", "sweep", "fp64", "soc", 30, 1, 1, 2, spin=True),
        # the reference's default run as its Fortran drives it: 4 x 3 x 3, one energy at a time
        _solve("sweep_ti_36", "sweep", "fp64", "ti_ref", 4, 3, 3, 3, sr_tol=1e-8),
        # the plain FP64 configuration: M = 64, 64 energies, site density and spin
        _solve("fp64_ti_64", "batch", "fp64", "ti", 20, 4, 4, 64, spin=True),
        # another channel of the reference at an odd size: a topological surface, 37 sites wide
        _solve("fp64_surface_74", "batch", "fp64", "surface", 25, 37, 1, 21),
        # superconducting contacts on a BdG Hamiltonian (8 orbitals a site, M = 72)
        _solve("fp64_bdg_72", "batch", "fp64", "ti", 9, 3, 3, 16, bdg=True),
        # the reference's production wire (10 x 10 x 8, M = 320), one rank's share of its 600 energies
        _solve("fp64_ti_320", "batch", "fp64", "ti", 10, 10, 8, 9, W=0.2),
        # the FP64 configuration at scale (M = 400): one energy, 4 disorder samples
        _solve("fp64_ti_400", "batch", "fp64", "ti", 24, 10, 10, 1, 4),
        # one serving request of the smallest cross-section, in the mixed form
        _solve("mixed_ti_144", "batch", "mixed", "ti", 75, 6, 6, 32),
        # an odd cross-section with every reduction a user can ask for
        _solve("mixed_ti_140_full", "batch", "mixed", "ti", 33, 5, 7, 11, 2, spin=True, currents=True),
        # the benchmark's wire in the mixed form: 8 energies x 4 disorder samples
        _solve("mixed_ti_400", "batch", "mixed", "ti", 100, 10, 10, 8, 4),
        # a biased wire of the self-consistent loop: the end slices differ, M = 576
        _solve("mixed_ti_576_bias", "batch", "mixed", "ti", 30, 12, 12, 2, 4, bias=True),
        # the electrostatics of the same loop: one grid per disorder sample
        dict(name="poisson_60x12x12", kind="poisson", npx=60, npy=12, npz=12, grids=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _flops(c):
    """Real flops of one pass: per slice and energy two inverses and four products of M x M
    complex blocks, per decimation iteration (18 of them) ten products and one inverse."""
    m = _m(c)
    per = 48.0 * m ** 3 * c["npx"] + 32.0 * m ** 3
    decimations = c["energies"] * (c["seeds"] * 2 if c["bias"] else 1)
    lead = 0.0 if c["bdg"] else (88.0 * 18 + 24.0) * m ** 3 * decimations
    return per * c["energies"] * c["seeds"] + lead


def _m(c):
    return NORB[c["model"]] * (2 if c["bdg"] else 1) * c["npy"] * c["npz"]


def draw(rng):
    kind = rng.choice(("sweep", "fp64", "fp64", "fp64", "mixed", "mixed", "mixed", "poisson"))
    if kind == "poisson":
        return dict(kind="poisson", npx=_log(rng, 9, 120), npy=rng.randint(3, 14), npz=rng.randint(3, 14),
                    grids=rng.randint(1, 8))
    while True:
        if kind == "sweep":
            model = rng.choice(("soc", "surface", "ti_ref", "ti"))
            wide = {"soc": 1, "surface": 12, "ti_ref": 4, "ti": 4}[model]
            npy = rng.randint(1, wide)
            npz = 1 if model in ("soc", "surface") else rng.randint(2, wide)
            c = _solve("", "sweep", "fp64", model, _log(rng, 4, 30), max(npy, 2) if model != "soc" else 1, npz,
                       rng.randint(1, 3), W=0.05)
            c["spin"] = model in ("ti", "soc") and rng.random() < 0.5
        else:
            model = rng.choice(("ti", "ti", "ti_ref", "surface")) if kind == "fp64" else "ti"
            if model == "surface":
                npy, npz = _log(rng, 5, 80), 1
            else:
                npy, npz = _log(rng, 2 if kind == "fp64" else 3, 12), _log(rng, 2 if kind == "fp64" else 3, 12)
            c = _solve("", "batch", kind, model, _log(rng, 4, 100), npy, npz, _log(rng, 1, 48), rng.choice((1, 1, 2, 4)),
                       W=0.1, bias=rng.random() < 0.25)
            c["spin"] = model in ("ti", "soc") and rng.random() < 0.5
            if kind == "mixed":
                c["currents"] = rng.random() < 0.3
            elif model == "ti" and npy * npz <= 16 and c["seeds"] == 1 and not c["bias"] and rng.random() < 0.3:
                c.update(bdg=True, spin=False)
        # at most the work, the memory and the chain of dependent steps of the listed cases
        m, items = _m(c), c["energies"] * c["seeds"]
        if _flops(c) <= (4e11 if c["form"] == "fp64" else 8e12) and 16.0 * m * m * c["npx"] * items <= 1.2e10 and \
                m * c["npx"] <= (9000 if c["form"] == "fp64" else 30000) and (kind != "sweep" or m * c["npx"] <= 1000):
            del c["name"]
            return c


def _inputs(c, seed):
    """Energies, occupations, weight, slots and the site potential of each disorder sample."""
    rng = np.random.default_rng(1000003 * seed + 17)
    lo, hi = WINDOW[c["model"]]
    grid = np.sort(rng.uniform(lo, hi, c["energies"]))
    e = np.repeat(grid, c["seeds"])
    slots = np.tile(np.arange(c["seeds"], dtype=np.int32), c["energies"])
    mid = 0.5 * (lo + hi)
    f1 = 1.0 / (1.0 + np.exp((e - mid - MU1) / KT))
    f2 = 1.0 / (1.0 + np.exp((e - mid - MU2) / KT))
    v = np.zeros((c["seeds"], c["npx"], c["npy"], c["npz"]))
    if c["npx"] > 2:
        v[:, 1:-1] = c["W"] * (rng.random((c["seeds"], c["npx"] - 2, c["npy"], c["npz"])) - 0.5)
    if c["bias"]:   # a potential drop along the wire, its own for each sample
        v += np.linspace(0.02, -0.02, c["npx"])[None, :, None, None] * (1.0 + 0.1 * rng.random((c["seeds"], 1, 1, 1)))
    flux = float(rng.uniform(0.3, 0.7)) if c["model"] == "ti" else 0.0
    return dict(e=e, f1=f1, f2=f2, dE=(hi - lo) / c["energies"], slots=slots, v=v, flux=flux)


def _model(c, flux, v):
    if c["model"] == "ti":
        return hamiltonian.wire_model(zeeman=0.01, flux=flux, V=v)
    if c["model"] == "ti_ref":
        return hamiltonian.wire_model(basis="reference", zeeman=0.01, V=v)
    t = {"surface": 3, "soc": 4}[c["model"]]
    return hamiltonian.channel_model(t, mu_t=0.0, V=v)


def prepare(case, seed):
    if case["kind"] == "poisson":
        rng = np.random.default_rng(1000003 * seed + 29)
        shape = (case["npx"], case["npy"], case["npz"], case["grids"])
        return dict(case=case, rho=np.asfortranarray(1e-3 * rng.standard_normal(shape)),
                    bc=(0.025, -0.025, 0.1), kappa=scf.kappa(100.0))
    c, q = case, _inputs(case, seed)
    norb = NORB[c["model"]] * (2 if c["bdg"] else 1)
    n = c["energies"] * c["seeds"]
    s = Solver(c["npx"], c["npy"], c["npz"], norb=norb, n_hamiltonians=c["seeds"], max_batch=1 if c["kind"] == "sweep" else n,
               eta=c["eta"], sr_tol=c["sr_tol"], calc_spin=c["spin"], precision=c["form"], calc_currents=c["currents"],
               contact_type=3 if c["bdg"] else 0)
    for k in range(c["seeds"]):
        if c["bdg"]:
            s.set_hamiltonian(*hamiltonian.bdg(*hamiltonian.ti_wire(c["npx"], c["npy"], c["npz"], zeeman=0.01, flux=q["flux"],
                                                                    disorder=q["v"][k]), c["npy"], c["npz"]), slot=k)
        else:
            s.build_hamiltonian(_model(c, q["flux"], q["v"][k]), slot=k)
    return dict(case=c, solver=s, **q)


def run(state):
    c = state["case"]
    if c["kind"] == "poisson":
        u, iters = scf.poisson_solve(state["rho"], state["bc"], state["kappa"])
        return dict(U=u, iters=iters)
    s = state["solver"]
    slots = None if c["kind"] == "sweep" else c["seeds"]
    rho_n, rho_p = s.new_site_array(slots), s.new_site_array(slots)
    spin = [s.new_site_array(slots) for _ in range(3)] if c["spin"] else None
    if c["kind"] == "sweep":
        cur, rows = np.zeros(2), []
        for e, f1, f2 in zip(state["e"], state["f1"], state["f2"]):
            rows.append(s.energy_sweep(e, f1, f2, state["dE"], rho_n, rho_p, cur, spin))
        out = {k: np.array([r[k] for r in rows]) for k in ("T12", "EDensity", "HDensity", "Modec1", "Modec2", "dosc",
                                                           "sr_status", "rgf_status")}
        out["contact_current"] = cur
    else:
        cur = [s.new_site_array(slots) for _ in range(3)] if c["currents"] else None
        out = s.solve_batch(state["e"], state["f1"], state["f2"], state["dE"], slots=state["slots"], rho_n=rho_n,
                            rho_p=rho_p, spin=spin, currents=cur)
        if cur:
            out.update(zip(("Jx", "Jy", "Jz"), cur))
    out.update(rho_n=rho_n, rho_p=rho_p)
    if spin:
        out.update(zip(("SigX", "SigY", "SigZ"), spin))
    return out


def work(case):
    if case["kind"] == "poisson":
        # about 90 conjugate-gradient steps of 21 operations a site; charge in, potential out
        n = case["npx"] * case["npy"] * case["npz"] * case["grids"]
        return dict(bytes=16.0 * n, flops=90.0 * 21 * n)
    m, sites = _m(case), case["npx"] * case["npy"] * case["npz"]
    return dict(bytes=16.0 * m * m * case["npx"] * case["seeds"] + 8.0 * 2 * sites * case["seeds"], flops=_flops(case))


# ---- the same results in plain 64-bit arithmetic -----------------------------------------
_S0, _SX, _SY = np.eye(2), np.array([[0, 1], [1, 0]], complex), np.array([[0, -1j], [1j, 0]])
_SZ = np.diag([1.0, -1.0]).astype(complex)


def _blocks(c):
    """On-site block and the three hops of the channel model, and its spin operators."""
    if c["model"] == "ti":
        tz = np.kron(_SZ, _S0)
        on = (0.3 - 1.5) * tz + 0.01 * np.kron(_S0, _SZ)
        hops = [0.25 * tz - 0.25j * np.kron(_SX, s) for s in (_SX, _SY, _SZ)]
    elif c["model"] == "ti_ref":
        g0 = np.diag([1.0, 1, -1, -1]).astype(complex)
        g = np.zeros((3, 4, 4), complex)
        g[0][[0, 1, 2, 3], [3, 2, 1, 0]] = [-1j, 1j, -1j, 1j]
        g[1][[0, 1, 2, 3], [3, 2, 1, 0]] = -1
        g[2][[0, 1, 2, 3], [2, 3, 0, 1]] = [-1j, -1j, 1j, 1j]
        on, hops = -1.5 * g0 + 0.01 * np.kron(_S0, _SZ), [0.5 * (g0 - 1j * x) for x in g]
    elif c["model"] == "surface":
        on, hops = np.zeros((2, 2), complex), [-0.5j * _SY, 0.5j * _SX, np.zeros((2, 2), complex)]
    else:
        on, hops = np.zeros((2, 2), complex), [-0.5j * _SY, np.zeros((2, 2), complex), np.zeros((2, 2), complex)]
    nh = on.shape[0]
    ops = [np.kron(np.eye(nh // 2), s) for s in (_SX, _SY, _SZ)]
    return on, hops, ops


def _slice(c, flux):
    """One slice without its potential, and the hop to the next one."""
    on, (hx, hy, hz), _ = _blocks(c)
    ny, nz, no = c["npy"], c["npz"], on.shape[0]
    h = np.zeros((nz, ny, no, nz, ny, no), complex)
    x = np.zeros_like(h)
    for z in range(nz):
        ph = np.exp(2j * math.pi * z * flux / ((ny - 1) * (nz - 1))) if flux and ny > 1 and nz > 1 else 1.0
        for y in range(ny):
            h[z, y, :, z, y], x[z, y, :, z, y] = on, hx
            if y + 1 < ny:
                h[z, y, :, z, y + 1], h[z, y + 1, :, z, y] = hy * ph, (hy * ph).conj().T
            if z + 1 < nz:
                h[z, y, :, z + 1, y], h[z + 1, y, :, z, y] = hz, hz.conj().T
    m = ny * nz * no
    return h.reshape(m, m), x.reshape(m, m)


def _decimate(alpha, hop, eta, tol):
    """Self-energy of a lead whose blocks couple through beta = -hop: (E, M, M) of alphas."""
    eye = torch.eye(alpha.shape[-1], dtype=alpha.dtype, device=alpha.device)
    g = torch.linalg.inv(alpha + 1j * eta * eye)
    t, tt = g @ hop.mH, g @ hop
    total, told = t.clone(), eye.expand_as(alpha).clone()
    busy = torch.ones(len(alpha), dtype=torch.bool, device=alpha.device)
    for _ in range(200):
        told = told @ tt
        w = torch.linalg.inv(eye - t @ tt - tt @ t)
        t, tt = w @ t @ t, w @ tt @ tt
        change = told @ t
        total = torch.where(busy[:, None, None], total + change, total)
        busy &= change.abs().amax((1, 2)) > tol
        if not busy.any():
            break
    return hop @ torch.linalg.inv(alpha - hop @ total) @ hop.mH


def exact(case, seed):
    if case["kind"] == "poisson":
        return None   # a whole number of iterations and the field they reach: no plain counterpart
    c, q = case, _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    h0, hx = _slice(c, q["flux"])
    no, nh = _blocks(c)[0].shape[0] * (2 if c["bdg"] else 1), _blocks(c)[0].shape[0]
    npx, ny, nz, m, n = c["npx"], c["npy"], c["npz"], _m(c), len(q["e"])
    diag = np.repeat(q["v"].transpose(0, 1, 3, 2).reshape(c["seeds"], npx, ny * nz), nh, axis=2)   # orbital order of a slice
    if c["bdg"]:
        electron = (np.arange(ny * nz)[:, None] * no + np.arange(nh)).ravel()

        def both(a):
            b = np.zeros((m, m), complex)
            b[np.ix_(electron, electron)], b[np.ix_(electron + nh, electron + nh)] = a, -a.conj()
            return b
        h0, hx = both(h0), both(hx)
        d2 = np.zeros((c["seeds"], npx, m))
        d2[:, :, electron], d2[:, :, electron + nh] = diag, -diag
        diag = d2
    h0, hx, diag = (torch.as_tensor(a, device=dev) for a in (h0, hx, diag))
    e, slots = torch.as_tensor(q["e"], device=dev), torch.as_tensor(q["slots"], device=dev).long()
    eye = torch.eye(m, dtype=h0.dtype, device=dev)

    def alpha(en, sl, x):
        return (en[:, None, None] + 1j * c["eta"]) * eye - h0 - torch.diag_embed(diag[sl, x]).to(h0.dtype)

    if c["bdg"]:
        gds = np.kron(np.eye(nh // 2), np.array([[0, 1], [-1, 0]]))
        sig = []
        for lead in (0, 1):
            ce = q["e"] + 1j * c["eta"]
            om, ph = 1.0 / np.sqrt(1e-6 - ce * ce), np.exp(0.8j) if lead == 0 else 1.0
            b = np.zeros((n, no, no), complex)
            b[:, :nh, :nh] = b[:, nh:, nh:] = (-om * ce)[:, None, None] * np.eye(nh)
            b[:, :nh, nh:], b[:, nh:, :nh] = (om * 1e-3 * ph)[:, None, None] * gds, (-om * 1e-3 * np.conj(ph))[:, None, None] * gds
            sig.append(torch.as_tensor(np.stack([np.kron(np.eye(ny * nz), x) for x in b]), device=dev))
    elif c["bias"]:
        sig = [_decimate(alpha(e, slots, x), h, c["eta"], c["sr_tol"]) for x, h in ((0, hx.mH), (npx - 1, hx))]
    else:   # the end slices carry no disorder: one lead per energy
        one = torch.as_tensor(q["e"][:: c["seeds"]].copy(), device=dev)
        a = alpha(one, torch.zeros(len(one), dtype=torch.long, device=dev), 0)
        sig = [_decimate(a, h, c["eta"], c["sr_tol"]).repeat_interleave(c["seeds"], 0) for h in (hx.mH, hx)]
    gam = [1j * (s - s.mH) for s in sig]
    dos = [-torch.diagonal(s, dim1=1, dim2=2).sum(1).imag / math.pi for s in sig]

    def w(x):
        a = alpha(e, slots, x)
        a = a - sig[0] if x == 0 else a
        return a - sig[1] if x == npx - 1 else a

    right = [None] * npx
    for x in reversed(range(npx)):
        right[x] = torch.linalg.inv(w(x) if x == npx - 1 else w(x) - hx @ right[x + 1] @ hx.mH)
    site = torch.zeros((2, npx, n, ny * nz, no, no), dtype=h0.dtype, device=dev)
    modes = [[None, None], [None, None]]
    g11 = right[0]
    g, left = None, None
    lefts = []
    for x in range(npx):
        g = right[0] if x == 0 else right[x] @ hx.mH @ g
        right[x] = None if x else right[0]
        left = torch.linalg.inv(w(x) if x == 0 else w(x) - hx.mH @ left @ hx)
        lefts.append(left)
        y = g @ gam[0]
        site[0, x] = torch.einsum("bsik,bsjk->bsij", y.reshape(n, ny * nz, no, m), g.conj().reshape(n, ny * nz, no, m))
        for k, at in enumerate((0, npx - 1)):
            if x == at:
                modes[k][0] = ((gam[k] @ y) * g.conj()).real.sum((1, 2))
    for x in reversed(range(npx)):
        g = lefts[x] if x == npx - 1 else lefts[x] @ hx @ g
        y = g @ gam[1]
        site[1, x] = torch.einsum("bsik,bsjk->bsij", y.reshape(n, ny * nz, no, m), g.conj().reshape(n, ny * nz, no, m))
        for k, at in enumerate((0, npx - 1)):
            if x == at:
                modes[k][1] = ((gam[k] @ y) * g.conj()).real.sum((1, 2))
    f1, f2 = (torch.as_tensor(q[k], device=dev)[None, :, None, None, None] for k in ("f1", "f2"))
    gn, gp = f1 * site[0] + f2 * site[1], (1 - f1) * site[0] + (1 - f2) * site[1]
    wgt = q["dE"] / (2 * math.pi)

    def sites(v):   # (npx, items, sites) -> the accumulated site array of each sample
        a = torch.zeros((npx, ny * nz, c["seeds"]), dtype=torch.float64, device=dev)
        a.index_add_(2, slots, wgt * v.permute(0, 2, 1))
        a = a.reshape(npx, nz, ny, c["seeds"]).permute(0, 2, 1, 3).cpu().numpy()
        return a[..., 0] if c["kind"] == "sweep" else a

    tr = lambda b, k: torch.diagonal(b, dim1=-2, dim2=-1).real[..., :k].sum(-1)  # noqa: E731
    t12 = modes[0][1]
    out = dict(EDensity=tr(gn, nh).sum((0, 2)) / (2 * math.pi), HDensity=tr(gp, nh).sum((0, 2)) / (2 * math.pi),
               Modec1=modes[0][0] + modes[0][1], Modec2=modes[1][0] + modes[1][1])
    if c["bdg"]:   # the supercurrent transmission, from the blocks of slice 1
        full = lambda b: torch.stack([torch.block_diag(*x) for x in b])  # noqa: E731
        a = 1j * full(gn[0]) @ sig[0].mH - g11 @ gam[0]
        sz = torch.as_tensor(np.where(np.arange(m) % no < nh, 1.0, -1.0), device=dev)
        t12 = (sz * torch.diagonal(a, dim1=1, dim2=2).real).sum(1)
    out["T12"] = t12
    out = {k: v.cpu().numpy() for k, v in out.items()}
    dos = [d.cpu().numpy() for d in dos]
    if c["kind"] == "sweep":
        qe, hp = 1.602e-19, 6.626e-34
        i = float((qe * q["dE"] / hp * out["T12"] * (q["f2"] - q["f1"])).sum())
        out.update(dosc=np.stack(dos, 1), sr_status=None, rgf_status=None, contact_current=np.array([i, -i]))
    else:
        out.update(DOSc1=dos[0], DOSc2=dos[1], status=None, sr_iters=None)
        if c["currents"]:
            out.update(Jx=None, Jy=None, Jz=None)   # sums of terms that are rounded to 32 bits
    out.update(rho_n=sites(tr(gn, no)), rho_p=sites(tr(gp, no)))
    if c["spin"]:
        for k, op in zip(("SigX", "SigY", "SigZ"), _blocks(c)[2]):
            out[k] = sites(torch.einsum("xbsij,ji->xbs", gn, torch.as_tensor(op.astype(complex), device=dev)).real)
    return out
