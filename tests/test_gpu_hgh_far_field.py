"""HGH local potential and its position gradient on both sides of the far-field switch.

Beyond 8 sqrt(2) r_loc (6 sqrt(2) r_loc in the FP32 force integral) only the Coulomb tail is evaluated.
The reference is the full formula in FP64 torch: each value is a handful of roundings (16 eps of the
largest term), the gradient a sum of N^3 of them whose roundings add as in the FP64 or float-float sums
of the kernels (FP32: each term carries a few 2^-24).
"""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def terms(grid, R, p):
    a = -grid.L / 2 + (torch.arange(grid.N, dtype=torch.float64, device="cuda") + 0.5) * grid.h
    X, Y, Z = torch.meshgrid(a, a, a, indexing="ij")
    d = (X - R[0], Y - R[1], Z - R[2])
    r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2 + 1e-30)
    q = (r / p.r_loc) ** 2
    c = p.c
    poly = c[0] + c[1] * q + c[2] * q ** 2 + c[3] * q ** 3
    dpoly = c[1] + 2 * c[2] * q + 3 * c[3] * q ** 2
    u = r / (math.sqrt(2.0) * p.r_loc)
    V = -p.Z_ion * torch.erf(u) / r + torch.exp(-0.5 * q) * poly
    f = 2 / math.sqrt(math.pi) * torch.exp(-u * u) / (math.sqrt(2.0) * p.r_loc * r) - torch.erf(u) / r ** 2
    dV = -p.Z_ion * f + torch.exp(-0.5 * q) * (dpoly - 0.5 * poly) * 2 * r / p.r_loc ** 2
    return V, [-dV * x / r for x in d]


# boxes that straddle the switch (2.3 bohr for H, 2.8 O, 4.6 Cl, 8.9 Li), odd and even grids, one centre
# close to a grid point
@pytest.mark.parametrize("symbols,N,L", [(("H",), 16, 4.0), (("O", "H"), 27, 9.0), (("Li", "Cl"), 33, 24.0),
                                          (("Cl",), 50, 11.0), (("O", "H", "H"), 1, 2.0)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
def test_local_potential_and_gradient(symbols, N, L, dtype):
    from gato_gb300.geometry import Nuclei
    from gato_gb300.grid import Grid3D
    from gato_gb300.pseudopotentials import hgh_local_grad, hgh_local_potential, lookup
    g = Grid3D(N, L)
    el = tuple(lookup(s) for s in symbols)
    pos = torch.tensor([[0.5 * g.h + 1e-9, 0.1, -0.2], [0.3, -0.7, 1.1], [-1.0, 0.4, 0.2]], dtype=torch.float64)[:len(el)]
    nuc = Nuclei(pos, torch.ones(len(el), dtype=torch.float64))
    gen = torch.Generator(device="cuda").manual_seed(N)
    rho = torch.rand(N, N, N, generator=gen, dtype=torch.float64, device="cuda").to(dtype)
    per = [terms(g, R, p) for R, p in zip(pos, el)]
    V = hgh_local_potential(nuc, el, g, dtype).double()
    ref, big = sum(v for v, _ in per), sum(v.abs() for v, _ in per)
    eps = 2.0 ** (-53 if dtype == torch.float64 else -24)
    peak = sum(abs(c) for p in el for c in p.c) + sum(p.Z_ion / p.r_loc for p in el)
    assert float(((V - ref).abs() / (big + 2.0 ** -29 * (dtype == torch.float32) + 1e-12 * peak)).max()) < 16 * eps + 1e-12
    got = hgh_local_grad(nuc, el, g, rho)
    want = torch.stack([torch.stack([(rho.double() * x).sum() for x in dv]) for _, dv in per]).cpu() * g.dV
    size = torch.stack([torch.stack([(rho.double() * x).abs().sum() for x in dv]) for _, dv in per]).cpu() * g.dV
    assert float(((got - want).abs() / size).max()) < 16 * eps
