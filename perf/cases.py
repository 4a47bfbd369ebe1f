"""Performance cases of the Fock-operator path, each through the package's public entry points.

Kinds of work (the ``kind`` of a case):

* ``hamiltonian``: ``Hamiltonian.apply`` and ``.rayleigh`` of one field, the single-particle layer.
* ``hartree``: ``hartree_potential`` of one density, once per SCF iteration.
* ``fock``: ``RHFFock.apply``, the matvec of the SCF eigensolver.
* ``block``: ``RHFFock.apply_block``, F phi_i for every occupied orbital with shared pair potentials.
* ``energy``: ``decompose_rhf_energy``, the five energy terms.
* ``force``: ``bo_grad_positions``, the Hellmann-Feynman forces at fixed orbitals.
* ``gradient``: ``bo_energy`` and its backward, the energy, the forces and dE/dphi of a geometry step.
* ``lanczos``: ``lanczos`` on a one-particle Hamiltonian, a whole eigensolve.
* ``imag``: ``imaginary_time``, the propagation of the hydrogen driver.
* ``scf``: ``scf_rhf``, a whole (short) self-consistent run.

Molecules are those of the drivers and the 48-system batch: ``water`` and ``hcl`` (four occupied
orbitals, HGH pseudopotentials), ``lih`` and ``helium`` (one orbital; HGH and softened Coulomb).
Spacings and boxes are the ones of the configurations (h = 0.25 bohr for water at 128^3, L = 12 in
the grid-convergence study). The ``exact`` side is plain torch in FP64: cuFFT convolutions, shifted
sums for the stencil, full-grid projectors.
"""
from __future__ import annotations

import math

import torch

from gato_gb300.geometry import Nuclei
from gato_gb300.grid import Grid3D
from gato_gb300.hamiltonian import Hamiltonian
from gato_gb300.physics.water import bo_energy, bo_grad_positions
from gato_gb300.potentials import softened_coulomb
from gato_gb300.pseudopotentials import hgh_local_potential, lookup, nonlocal_for
from gato_gb300.scf import RHFFock, decompose_rhf_energy, from_fields, scf_rhf
from gato_gb300.solvers.imag_time import imaginary_time
from gato_gb300.solvers.lanczos import default_krylov_dim, lanczos
from gato_gb300.solvers.poisson import hartree_potential

DTYPES = {"f64": torch.float64, "f32": torch.float32}
N_OCC = {"water": 4, "hcl": 4, "lih": 1, "helium": 1}
SYMBOLS = {"water": ("O", "H", "H"), "hcl": ("H", "Cl"), "lih": ("Li", "H")}

# Published HGH (1998) LDA parameters, for the exact side: Z_ion, r_loc, c, ((l, r_l, h), ...)
HGH = {
    "H": (1.0, 0.2, (-4.0663326, 0.6778322), ()),
    "O": (6.0, 0.24762086, (-16.5803180, 2.39570952), ((0, 0.22178614, ((18.26691718,),)),)),
    "Li": (1.0, 0.78755305, (-1.89261247, 0.28605968),
           ((0, 0.66637518, ((1.85881111,),)), (1, 1.07930561, ((-0.00589504,),)))),
    "Cl": (7.0, 0.41, (-6.86475431,),
           ((0, 0.33820832, ((9.06223968, -1.96193036), (-1.96193036, 5.06568240))),
            (1, 0.37613709, ((4.46587640,),)))),
}


def _case(kind, N, L, dtype, **kw):
    c = {"kind": kind, "N": int(N), "L": float(L), "dtype": dtype}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: one particle in a potential on a test-sized grid; launches and host time are all of it
        dict(_case("hamiltonian", 16, 8.0, "f64", order=2, boundary="dirichlet"), name="hamiltonian_16_f64"),
        # the Hartree solve of every iteration of the helium run, in the default precision
        dict(_case("hartree", 96, 16.0, "f64"), name="hartree_96_f64"),
        # water in the L = 12 box of the grid-convergence study, mixed precision: a small Fock matvec
        dict(_case("fock", 40, 12.0, "f32", molecule="water"), name="fock_40_f32"),
        # a box study's odd-sized grid (L = 10, h = 0.1), default precision
        dict(_case("fock", 100, 10.0, "f64", molecule="water"), name="fock_100_f64"),
        # the matvec of the 128^3 water run in mixed precision: half of every SCF iteration
        dict(_case("fock", 128, 32.0, "f32", molecule="water"), name="fock_128_f32"),
        # the benchmark's step: F phi_i for the four orbitals of water at 128^3, ten pair solves
        dict(_case("block", 128, 32.0, "f32", molecule="water"), name="block_128_f32"),
        # the largest grid of the batch: HCl at 160^3
        dict(_case("block", 160, 38.4, "f32", molecule="hcl"), name="block_160_f32"),
        # the FP64 energy of every late iteration of a mixed SCF
        dict(_case("energy", 128, 32.0, "f64", molecule="water"), name="energy_128_f64"),
        # forces of a mixed-precision geometry step
        dict(_case("force", 128, 32.0, "f32", molecule="water"), name="force_128_f32"),
        # energy, forces and orbital gradient through autograd, default precision
        dict(_case("gradient", 64, 16.0, "f64", molecule="water"), name="gradient_64_f64"),
        # the hydrogen configuration in mixed precision: 80 Krylov steps on 64^3, 7-point Laplacian
        dict(_case("lanczos", 64, 20.0, "f32", order=2, m=80, K=1), name="lanczos_64_f32"),
        # a whole run, two SCF iterations of the helium driver at its default size and precision; a mixed run
        # is made of the f32 matvec, f64 energy and f64 Hartree calls above
        dict(_case("scf", 64, 10.0, "f64", molecule="helium", iters=2), name="scf_64_f64"),
    ]


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _size(rng, lo, hi, poisson=True):
    """Log-uniform in [lo, hi]: half the draws on the batch's and studies' grids, the rest anywhere, odd ones among them."""
    if rng.random() < 0.5:
        return rng.choice([n for n in (24, 32, 40, 48, 64, 80, 96, 128, 160) if lo <= n <= hi])
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if lo <= n <= hi and (not poisson or _smooth(n)):
            return n


def draw(rng):
    kind = rng.choice(["hamiltonian", "hartree", "fock", "fock", "block", "block", "energy", "force",
                       "gradient", "lanczos", "imag", "scf"])
    dtype = rng.choice(["f64", "f32"])
    h = round(rng.uniform(0.2, 0.3), 4)
    mol = rng.choice(["water", "hcl", "lih", "helium"])
    if kind == "hamiltonian":
        n = _size(rng, 12, 160, poisson=False)
        return _case(kind, n, n * h, dtype, order=rng.choice([2, 4]), boundary=rng.choice(["dirichlet", "periodic"]))
    if kind == "hartree":
        n = _size(rng, 16, 160 if dtype == "f32" else 128)
        return _case(kind, n, n * h, dtype)
    if kind in ("fock", "block"):
        n = _size(rng, 20, 160 if dtype == "f32" else 96)
        return _case(kind, n, n * h, dtype, molecule=mol)
    if kind == "energy":
        n = _size(rng, 20, 128)
        return _case(kind, n, n * h, "f64", molecule=mol)
    if kind == "force":
        n = _size(rng, 20, 160 if dtype == "f32" else 128)
        return _case(kind, n, n * h, dtype, molecule=rng.choice(["water", "hcl", "lih"]))
    if kind == "gradient":
        n = _size(rng, 20, 80)
        return _case(kind, n, n * h, "f64", molecule=rng.choice(["water", "hcl", "lih"]))
    if kind == "lanczos":
        n = _size(rng, 20, 64, poisson=False)
        return _case(kind, n, n * h, dtype, order=rng.choice([2, 4]), m=rng.choice([40, 60, 80]), K=1)
    if kind == "imag":
        n = _size(rng, 20, 96, poisson=False)
        return _case(kind, n, n * h, "f64", order=rng.choice([2, 4]), steps=rng.choice([50, 100, 200]))
    mol = rng.choice(["water", "helium"])
    n = _size(rng, 28, 50 if mol == "water" else 64)
    return _case(kind, n, n * h, "f64", molecule=mol, iters=1)


# ---- inputs ------------------------------------------------------------------------------------

def _coords(N, L):
    a = -L / 2 + (torch.arange(N, dtype=torch.float64, device="cuda") + 0.5) * (L / N)
    return torch.meshgrid(a, a, a, indexing="ij")


def _rand(seed):
    g = torch.Generator(device="cpu")
    g.manual_seed(int(seed) * 7919 + 11)
    return g


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, dtype=torch.float64)


def _positions(mol, g):
    """(K, 3) positions: the drivers' geometries with the configurations' +-0.05 bohr jitter."""
    half = math.radians(104.5) / 2
    base = {"water": [[0.0, 0.0, 0.0], [1.81 * math.sin(half), 0.0, 1.81 * math.cos(half)],
                      [-1.81 * math.sin(half), 0.0, 1.81 * math.cos(half)]],
            "hcl": [[0.0, 0.0, -1.2], [0.0, 0.0, 1.2]],
            "lih": [[0.0, 0.0, -1.5], [0.0, 0.0, 1.5]],
            "helium": [[0.0, 0.0, 0.0]]}[mol]
    p = torch.tensor(base, dtype=torch.float64)
    return p + _uniform(g, -0.05, 0.05, *p.shape)


def _noise(seed, N):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 104729 + 5)
    return torch.randn(N, N, N, generator=g, dtype=torch.float64, device="cuda")


def _orbitals(pos, n, N, L, g, seed, dtype):
    """n orthonormal orbitals: Gaussians of seeded width around the nuclei times a seeded linear factor."""
    X, Y, Z = _coords(N, L)
    dV = (L / N) ** 3
    orb = torch.empty(n, N, N, N, dtype=torch.float64, device="cuda")
    noise = _noise(seed, N)
    for k in range(n):
        c = pos[k % len(pos)] + _uniform(g, -0.3, 0.3, 3)
        al = float(_uniform(g, 0.4, 0.9, 1))
        w = _uniform(g, -0.3, 0.3, 3)
        env = torch.exp(-al * ((X - c[0]) ** 2 + (Y - c[1]) ** 2 + (Z - c[2]) ** 2))
        orb[k] = env * (1.0 + w[0] * X + w[1] * Y + w[2] * Z + 1e-3 * noise)
    for i in range(n):
        for j in range(i):
            orb[i] -= (orb[i] * orb[j]).sum() * dV * orb[j]
        orb[i] /= torch.sqrt((orb[i] ** 2).sum() * dV)
    return orb.to(dtype).contiguous()


def _vh(N, L, n_el, dtype):
    """The Hartree potential of n_el electrons in one Gaussian charge of width 1.2 bohr."""
    X, Y, Z = _coords(N, L)
    r = torch.sqrt(X * X + Y * Y + Z * Z + 1e-12)
    return (n_el * torch.erf(r / 1.2) / r).to(dtype).contiguous()


def _inputs(case, seed):
    """Everything the seed decides, by plain torch alone (both ``prepare`` and ``exact`` start from it)."""
    N, L, kind = case["N"], case["L"], case["kind"]
    dtype = DTYPES[case["dtype"]]
    g = _rand(seed)
    d = {"N": N, "L": L, "h": L / N, "dtype": dtype}
    if kind in ("hamiltonian", "imag"):
        # softened Coulomb centre near the origin and a smooth start with a little noise
        X, Y, Z = _coords(N, L)
        d["center"] = [float(v) for v in _uniform(g, -0.2, 0.2, 3)]
        w = _uniform(g, -0.2, 0.2, 3)
        psi = torch.exp(-0.5 * (X * X + Y * Y + Z * Z)) * (1.0 + w[0] * X + w[1] * Y + w[2] * Z)
        d["psi"] = (psi + 1e-3 * torch.exp(-0.2 * (X * X + Y * Y + Z * Z)) * _noise(seed, N)).to(dtype).contiguous()
    elif kind == "lanczos":
        # the hydrogen configuration: a uniform random start vector
        gg = torch.Generator(device="cuda")
        gg.manual_seed(int(seed) * 31337 + 3)
        d["center"] = [float(v) for v in _uniform(g, -0.2, 0.2, 3)]
        d["psi"] = torch.rand(N, N, N, generator=gg, dtype=torch.float64, device="cuda").to(dtype)
    elif kind == "hartree":
        pos = _positions("water", g)
        orb = _orbitals(pos, 4, N, L, g, seed, torch.float64)
        d["rho"] = (2.0 * (orb * orb).sum(0)).to(dtype).contiguous()
    else:
        mol = case["molecule"]
        d["mol"], d["n"] = mol, N_OCC[mol]
        d["pos"] = _positions(mol, g)
        d["orb"] = _orbitals(d["pos"], d["n"], N, L, g, seed, dtype)
        if kind in ("fock", "block"):
            d["vh"] = _vh(N, L, 2 * d["n"], dtype)
        if kind == "fock":
            psi = d["orb"].double().sum(0)
            psi = psi + 0.05 * psi.abs().sqrt() * _noise(seed + 1, N)
            d["psi"] = (psi / torch.sqrt((psi * psi).sum() * d["h"] ** 3)).to(dtype).contiguous()
    return d


def _charges(mol):
    return torch.tensor({"water": [8.0, 1.0, 1.0], "hcl": [1.0, 17.0], "lih": [3.0, 1.0], "helium": [2.0]}[mol],
                        dtype=torch.float64)


def prepare(case, seed):
    d = _inputs(case, seed)
    kind, dtype = case["kind"], d["dtype"]
    grid = Grid3D(d["N"], d["L"])
    s = {"kind": kind, "grid": grid}
    if kind in ("hamiltonian", "imag", "lanczos"):
        V = softened_coulomb(grid, 1.0, 0.1 if kind == "lanczos" else None, d["center"], dtype=dtype)
        s["H"] = Hamiltonian(grid, V, case.get("boundary", "dirichlet"), case["order"])
        s["psi"] = d["psi"]
        s["m"], s["K"], s["steps"] = case.get("m"), case.get("K"), case.get("steps")
        return s
    if kind == "hartree":
        s["rho"] = d["rho"]
        return s
    mol = d["mol"]
    nuc = Nuclei(d["pos"], _charges(mol))
    s["orb"], s["n"] = from_fields(d["orb"]), d["n"]
    if kind in ("force", "gradient"):
        s["pos"], s["charges"], s["elements"] = d["pos"], nuc.charges, tuple(lookup(e) for e in SYMBOLS[mol])
        return s
    vdtype = torch.float64 if kind == "scf" else dtype
    if mol == "helium":
        s["V"], s["nl"] = softened_coulomb(grid, 2.0, None, tuple(float(v) for v in d["pos"][0]), dtype=vdtype), None
    else:
        el = tuple(lookup(e) for e in SYMBOLS[mol])
        s["V"], s["nl"] = hgh_local_potential(nuc, el, grid, vdtype), nonlocal_for(nuc, el, grid, dtype)
    if kind in ("fock", "block"):
        s["F"] = RHFFock(grid, s["V"], s["orb"], d["vh"], order=4, V_nl_apply=s["nl"])
        s["psi"] = d.get("psi")
    if kind == "scf":
        s["precision"], s["iters"] = ("mixed" if case["dtype"] == "f32" else "fp64"), case["iters"]
    return s


def run(s):
    kind, grid = s["kind"], s["grid"]
    if kind == "hamiltonian":
        return {"Hpsi": s["H"].apply(s["psi"]), "rayleigh": s["H"].rayleigh(s["psi"])}
    if kind == "hartree":
        return {"J": hartree_potential(s["rho"], grid)}
    if kind == "fock":
        return {"Fpsi": s["F"].apply(s["psi"])}
    if kind == "block":
        return {"Fphi": s["F"].apply_block()}
    if kind == "energy":
        t = decompose_rhf_energy(s["orb"], s["V"], grid, order=4, V_nl_apply=s["nl"])
        return {"kinetic": t.kinetic, "v_ext": t.v_ext, "v_nl": t.v_nl, "hartree": t.hartree, "exchange": t.exchange}
    if kind == "force":
        return {"dE_dR": bo_grad_positions(s["pos"], s["charges"], s["orb"], s["elements"], grid)}
    if kind == "gradient":
        p = s["pos"].clone().requires_grad_(True)
        orb = s["orb"].detach().requires_grad_(True)
        E = bo_energy(p, s["charges"], orb, s["elements"], grid)
        E.backward()
        return {"E": E.detach(), "dE_dR": p.grad, "dE_dphi": orb.grad}
    if kind == "lanczos":
        r = lanczos(s["H"], s["psi"], n_iters=s["m"], n_eigenstates=s["K"])
        return {"eigenvalues": r.eigenvalues, "eigenstates": r.eigenstates}
    if kind == "imag":
        psi, hist = imaginary_time(s["H"], s["psi"], n_steps=s["steps"], log_every=50)
        return {"psi": psi, "energies": hist.energies}
    r = scf_rhf(s["V"], grid, s["n"], initial_orbitals=s["orb"], max_iters=s["iters"], mixing=0.5, order=4,
                V_nl_apply=s["nl"], precision=s["precision"])
    return {"orbitals": r.orbitals, "energy": r.energy, "orbital_energies": r.orbital_energies,
            "history": r.energy_history}


def _solve_flops(N):
    """One real pair potential: half a complex convolution on the doubled grid, zero halves skipped."""
    M = 2 * N
    return 0.5 * 2 * (N * N + N * M + M * M) * 5.0 * M * (math.log2(M) - 1)


def work(case):
    N, n3, s = case["N"], case["N"] ** 3, 8 if case["dtype"] == "f64" else 4
    kind, sten = case["kind"], (30 if case.get("order", 4) == 4 else 16)
    n = N_OCC.get(case.get("molecule"), 1)
    pairs = n * (n + 1) // 2
    if kind == "hamiltonian":
        return {"bytes": 3 * n3 * s, "flops": (2 * sten + 6) * n3}
    if kind == "hartree":
        return {"bytes": 2 * n3 * s, "flops": _solve_flops(N)}
    if kind == "fock":
        return {"bytes": (n + 3) * n3 * s, "flops": n * (_solve_flops(N) + 3 * n3) + sten * n3}
    if kind == "block":
        return {"bytes": (2 * n + 1) * n3 * s, "flops": pairs * (_solve_flops(N) + 4 * n3) + n * sten * n3}
    if kind == "energy":
        # a spectral sum needs the forward half of each solve only
        return {"bytes": (n + 1) * n3 * s, "flops": (pairs + 1) * _solve_flops(N) / 2 + n * (sten + 6) * n3}
    if kind == "force":
        return {"bytes": n * n3 * s, "flops": (2 * n + 40) * n3}
    if kind == "gradient":
        return {"bytes": 2 * n * n3 * s, "flops": (pairs + 2) * 1.5 * _solve_flops(N) + 2 * n * sten * n3}
    if kind == "lanczos":
        m = case["m"]
        return {"bytes": (m * (m + 1) / 2 + 4 * m) * n3 * s, "flops": (2 * m * (m + 1) + sten * m) * n3}
    if kind == "imag":
        return {"bytes": 3 * n3 * s * case["steps"], "flops": (sten + 4) * n3 * case["steps"]}
    m = default_krylov_dim(N, n)
    per = {"bytes": (m * (m + 1) / 2 + (n + 4) * m) * n3 * s,
           "flops": m * (n * _solve_flops(N) + sten * n3) + 2 * m * (m + 1) * n3 + (pairs + 3) * _solve_flops(N)}
    return {k: v * case["iters"] for k, v in per.items()}


# ---- the same results in plain torch, 64 bits ----------------------------------------------------

def _lap(psi, h, order, boundary="dirichlet"):
    cf = {2: (-6.0, (1.0,)), 4: (3 * (-30.0 / 12.0), (16.0 / 12.0, -1.0 / 12.0))}[order]
    out = cf[0] * psi
    for ax in (-3, -2, -1):
        n = psi.shape[ax]
        for d, c in enumerate(cf[1], start=1):
            if boundary == "periodic":
                out = out + c * (torch.roll(psi, d, ax) + torch.roll(psi, -d, ax))
            elif n > d:
                out.narrow(ax, d, n - d).add_(psi.narrow(ax, 0, n - d), alpha=c)
                out.narrow(ax, 0, n - d).add_(psi.narrow(ax, d, n - d), alpha=c)
    return out / (h * h)


class _Hockney:
    def __init__(self, N, h, eps):
        M = 2 * N
        i = torch.arange(M, device="cuda", dtype=torch.float64)
        x = torch.where(i < N, i, i - M) * h
        r2 = (x * x)[:, None, None] + (x * x)[None, :, None] + (x * x)[None, None, :]
        self.G = torch.fft.rfftn(1.0 / torch.sqrt(r2 + eps * eps)).real * h ** 3
        self.N, self.M = N, M

    def __call__(self, rho):
        N, M = self.N, self.M
        f = torch.fft.rfftn(rho, s=(M, M, M))
        return torch.fft.irfftn(f * self.G, s=(M, M, M))[:N, :N, :N].contiguous()


def _soft(N, L, Z, eps, center):
    X, Y, Z0 = _coords(N, L)
    return -Z / torch.sqrt((X - center[0]) ** 2 + (Y - center[1]) ** 2 + (Z0 - center[2]) ** 2 + eps * eps)


def _vloc(mol, pos, N, L, rho=None):
    """V_loc of the molecule, and with rho the (K, 3) derivatives of int rho V_loc."""
    X, Y, Z0 = _coords(N, L)
    V, grads = 0.0, []
    for e, R in zip(SYMBOLS[mol], pos):
        Zi, rl, c, _ = HGH[e]
        d = (X - R[0], Y - R[1], Z0 - R[2])
        r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2 + 1e-30)
        q = (r / rl) ** 2
        poly = sum(ck * q ** k for k, ck in enumerate(c))
        V = V - Zi * torch.erf(r / (math.sqrt(2.0) * rl)) / r + torch.exp(-0.5 * q) * poly
        if rho is not None:
            u = r / (math.sqrt(2.0) * rl)
            de = -Zi * (2.0 / math.sqrt(math.pi) * torch.exp(-u * u) / (math.sqrt(2.0) * rl * r) - torch.erf(u) / r ** 2)
            dpoly = sum(k * ck * q ** (k - 1) for k, ck in enumerate(c) if k > 0) if len(c) > 1 else 0.0
            dv = de + torch.exp(-0.5 * q) * (dpoly - 0.5 * poly) * 2.0 * r / (rl * rl)
            grads.append(torch.stack([(-rho * dv * dk / r).sum() * (L / N) ** 3 for dk in d]))
    return V if rho is None else (V, torch.stack(grads).cpu())


def _projectors(mol, pos, N, L):
    """[(atom, h matrix, [(value, gradient in r)] per radial index)] of every (channel, m)."""
    X, Y, Z0 = _coords(N, L)
    out = []
    for a, (e, R) in enumerate(zip(SYMBOLS[mol], pos)):
        for ell, rl, hm in HGH[e][3]:
            d = (X - R[0], Y - R[1], Z0 - R[2])
            r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
            for m in range(2 * ell + 1):
                ps = []
                for i in range(1, len(hm) + 1):
                    nn = ell + (4.0 * i - 1.0) / 2.0
                    norm = math.sqrt(2.0) / (rl ** nn * math.sqrt(math.gamma(nn)))
                    ylm = 1.0 / math.sqrt(4 * math.pi) if ell == 0 else math.sqrt(3.0 / (4 * math.pi))
                    ang = 1.0 if ell == 0 else d[(1, 2, 0)[m]]   # r Y_1m is linear in the coordinate
                    rad = norm * ylm * r2 ** (i - 1) * torch.exp(-r2 / (2 * rl * rl))
                    p = rad * ang
                    # dp/dd_c of rad(r2) * ang
                    drad = norm * ylm * torch.exp(-r2 / (2 * rl * rl)) * (
                        ((2 * (i - 1)) * r2 ** (i - 2) if i > 1 else 0.0) - r2 ** (i - 1) / (rl * rl))
                    gr = [drad * dc * ang + (rad if (ell == 1 and c == (1, 2, 0)[m]) else 0.0) for c, dc in enumerate(d)]
                    ps.append((p, gr))
                out.append((a, torch.tensor(hm, dtype=torch.float64, device="cuda"), ps))
    return out


def _vnl(projs, psi, dV):
    out = torch.zeros_like(psi)
    for _, hm, ps in projs:
        c = hm @ torch.stack([(p * psi).sum() * dV for p, _ in ps])
        for ci, (p, _) in zip(c, ps):
            out += ci * p
    return out


def _system(case, d, vdtype):
    """(V_ext as the run is given it, projectors) in FP64."""
    N, L, mol = d["N"], d["L"], d["mol"]
    if mol == "helium":
        return _soft(N, L, 2.0, d["h"] / 2, d["pos"][0]).to(vdtype).double(), []
    return _vloc(mol, d["pos"], N, L).to(vdtype).double(), _projectors(mol, d["pos"], N, L)


def _fock(psi, orb, V, projs, hock, h):
    out = -0.5 * _lap(psi, h, 4) + V * psi + _vnl(projs, psi, h ** 3)
    for phi in orb:
        out -= phi * hock(phi * psi)
    return out


def _energy(orb, V, projs, hock, h):
    dV = h ** 3
    rho = 2.0 * (orb * orb).sum(0)
    t = [2 * sum((p * (-0.5 * _lap(p, h, 4))).sum() for p in orb) * dV,
         2 * sum((p * V * p).sum() for p in orb) * dV,
         2 * sum((p * _vnl(projs, p, dV)).sum() for p in orb) * dV,
         0.5 * (rho * hock(rho)).sum() * dV]
    ex = 0.0
    for i in range(len(orb)):
        for j in range(i, len(orb)):
            pij = orb[i] * orb[j]
            ex = ex - (1.0 if i == j else 2.0) * (pij * hock(pij)).sum() * dV
    return [torch.as_tensor(v, dtype=torch.float64) for v in t + [ex]]


def _lanczos(apply, psi0, m, K, dV):
    """m steps with two Gram-Schmidt passes; Ritz vectors with their largest tridiagonal component positive."""
    shape, n = psi0.shape, psi0.numel()
    V = torch.zeros(m + 1, n, dtype=torch.float64, device="cuda")
    V[0] = psi0.reshape(-1) / torch.sqrt((psi0 * psi0).sum() * dV)
    al, be = [], []
    for j in range(m):
        w = apply(V[j].reshape(shape)).reshape(-1)
        a = (V[j] @ w) * dV
        w = w - a * V[j] - (be[-1] * V[j - 1] if j else 0.0)
        for _ in range(2):
            w = w - (V[:j + 1] @ w * dV) @ V[:j + 1]
        b = torch.sqrt((w @ w) * dV)
        V[j + 1] = w / b
        al.append(a)
        be.append(b)
    T = torch.diag(torch.stack(al)) + torch.diag(torch.stack(be[:-1]), 1) + torch.diag(torch.stack(be[:-1]), -1)
    lam, Y = torch.linalg.eigh(T.cpu())
    Y = Y[:, :K]
    Y = Y * torch.sign(Y.gather(0, Y.abs().argmax(0, keepdim=True)))
    return lam[:K], (Y.T.cuda() @ V[:m]).reshape(K, *shape)


def exact(case, seed):
    d = _inputs(case, seed)
    N, L, h, kind = d["N"], d["L"], d["h"], case["kind"]
    dV = h ** 3
    if kind in ("hamiltonian", "imag", "lanczos"):
        V = _soft(N, L, 1.0, 0.1 if kind == "lanczos" else h / 2, d["center"]).to(d["dtype"]).double()
        psi = d["psi"].double()
        ap = lambda p: -0.5 * _lap(p, h, case["order"], case.get("boundary", "dirichlet")) + V * p   # noqa: E731
        if kind == "hamiltonian":
            hp = ap(psi)
            return {"Hpsi": hp, "rayleigh": (psi * hp).sum() / (psi * psi).sum()}
        if kind == "lanczos":
            lam, X = _lanczos(ap, psi, case["m"], case["K"], dV)
            return {"eigenvalues": lam, "eigenstates": X.permute(1, 2, 3, 0)}
        e = []
        psi = psi / torch.sqrt((psi * psi).sum() * dV)
        for i in range(case["steps"]):
            psi = psi - (h * h / 10.0) * ap(psi)
            psi = psi / torch.sqrt((psi * psi).sum() * dV)
            if i % 50 == 0 or i == case["steps"] - 1:
                e.append(float((psi * ap(psi)).sum() / (psi * psi).sum()))
        return {"psi": psi, "energies": e}
    hock = _Hockney(N, h, h / 2)
    if kind == "hartree":
        return {"J": hock(d["rho"].double())}
    orb = d["orb"].double()
    if kind == "force":
        return {"dE_dR": _forces(case, d, orb)}
    V, projs = _system(case, d, torch.float64 if kind == "scf" else d["dtype"])
    if kind == "fock":
        return {"Fpsi": _fock(d["psi"].double(), orb, V + d["vh"].double(), projs, hock, h)}
    if kind == "block":
        F = torch.stack([_fock(p, orb, V + d["vh"].double(), projs, hock, h) for p in orb])
        return {"Fphi": F}
    if kind == "energy":
        return dict(zip(("kinetic", "v_ext", "v_nl", "hartree", "exchange"), _energy(orb, V, projs, hock, h)))
    if kind == "gradient":
        Vh = hock(2.0 * (orb * orb).sum(0))
        g = torch.stack([_fock(p, orb, V + Vh, projs, hock, h) for p in orb]) * (4.0 * dV)
        Zi = [HGH[e][0] for e in SYMBOLS[d["mol"]]]
        enn = sum(Zi[a] * Zi[b] / torch.linalg.norm(d["pos"][a] - d["pos"][b])
                  for a in range(len(Zi)) for b in range(a + 1, len(Zi)))
        E = sum(t.cpu() for t in _energy(orb, V, projs, hock, h)) + enn
        return {"E": E, "dE_dR": _forces(case, d, orb), "dE_dphi": g.permute(1, 2, 3, 0)}
    return _scf(case, d, orb, V, projs, hock, h)


def _forces(case, d, orb):
    N, L, mol, pos = d["N"], d["L"], d["mol"], d["pos"]
    dV = d["h"] ** 3
    _, g = _vloc(mol, pos, N, L, rho=2.0 * (orb * orb).sum(0))
    for a, hm, ps in _projectors(mol, pos, N, L):
        for phi in orb:
            ov = torch.stack([(p * phi).sum() * dV for p, _ in ps])
            c = hm @ ov
            for ci, (_, gr) in zip(c, ps):
                for k in range(3):
                    g[a, k] += float(4.0 * ci * (-(gr[k] * phi).sum() * dV))
    Zi = [HGH[e][0] for e in SYMBOLS[mol]]
    for a in range(len(Zi)):
        for b in range(len(Zi)):
            if a != b:
                r = pos[a] - pos[b]
                g[a] -= Zi[a] * Zi[b] * r / torch.linalg.norm(r) ** 3
    return g


def _scf(case, d, orb, V, projs, hock, h):
    n, N, dV = d["n"], d["N"], h ** 3
    m = default_krylov_dim(N, n)
    rho, hist = 2.0 * (orb * orb).sum(0), []
    for _ in range(case["iters"]):
        Vt = V + hock(rho)
        lam, new = _lanczos(lambda p: _fock(p, orb, Vt, projs, hock, h), orb.sum(0), m, n, dV)
        orb = new
        rho = 0.5 * (2.0 * (orb * orb).sum(0)) + 0.5 * rho
        hist.append(float(sum(_energy(orb, V, projs, hock, h))))
    return {"orbitals": orb.permute(1, 2, 3, 0), "energy": hist[-1], "orbital_energies": lam, "history": hist}
