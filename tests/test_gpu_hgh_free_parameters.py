"""HGH local parts with parameters no element has: where the Gaussian terms reach past the far-field switch
(large coefficients, no ion charge) they count there too, and parameters that are not finite or have r_loc < 0
give what the formula gives, everywhere.

A value is a handful of roundings and an exponential whose argument q / 2, q = (r / r_loc)^2, carries a few more:
16 (1 + q) eps of the magnitudes of its two terms, beside the smallest subnormals; a coordinate -L/2 + (i + 1/2) h
carries 2 eps L of FP64 on either side, which the terms' slopes carry on. Forces are taken on a density that is zero
inside the switch.
"""
import math

import pytest
import torch

from test_gpu_hgh_far_field import terms

pytestmark = pytest.mark.gpu

PARAMS = {"large": (1.0, 0.3, (0.0, 0.0, 0.0, 1e10)), "uncharged": (0.0, 0.3, (1.0, 0.0, 0.0, 1.0)),
          "negative": (2.0, -0.3, (1.0, 0.5, 0.0, 0.0)), "nan": (2.0, 0.3, (math.nan, 0.0, 0.0, 0.0)),
          "inf": (2.0, 0.3, (0.0, math.inf, 0.0, 0.0))}


@pytest.mark.parametrize("kind", list(PARAMS))
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
def test_free_parameters(kind, dtype):
    from gato_gb300.geometry import Nuclei
    from gato_gb300.grid import Grid3D
    from gato_gb300.pseudopotentials import HGHParams, hgh_local_grad, hgh_local_potential
    g = Grid3D(40, 9.0)
    p = HGHParams("X", *PARAMS[kind])
    R = torch.tensor([[0.1, -0.2, 0.05]], dtype=torch.float64)
    nuc = Nuclei(R, torch.ones(1, dtype=torch.float64))
    V, dV = terms(g, R[0], p)
    a = -g.L / 2 + (torch.arange(g.N, dtype=torch.float64, device="cuda") + 0.5) * g.h
    X, Y, Z = torch.meshgrid(a, a, a, indexing="ij")
    q = ((X - R[0, 0]) ** 2 + (Y - R[0, 1]) ** 2 + (Z - R[0, 2]) ** 2) / p.r_loc ** 2
    eps, tiny = (2.0 ** -53, 2.0 ** -1060) if dtype == torch.float64 else (2.0 ** -24, 2.0 ** -149)
    got = hgh_local_potential(nuc, [p], g, dtype).double()
    nan = torch.isnan(V)
    assert torch.equal(torch.isnan(got), nan)
    assert torch.equal(torch.isinf(got), torch.isinf(V))
    ok = torch.isfinite(V)
    r, c, gauss = q.sqrt() * abs(p.r_loc), [abs(x) for x in p.c], torch.exp(-0.5 * q)
    tail = p.Z_ion * torch.erf(r / (math.sqrt(2.0) * abs(p.r_loc))) / r
    poly, dpoly = c[0] + q * (c[1] + q * (c[2] + q * c[3])), c[1] + q * (2 * c[2] + q * 3 * c[3])
    size, slope = tail + gauss * poly, 2 * tail / r + gauss * (dpoly + 0.5 * poly) * 2 * r / p.r_loc ** 2
    bound = 16 * (1 + q) * eps * size + 4 * 2.0 ** -53 * g.L * slope + tiny
    assert ((got - V).abs()[ok] <= bound[ok]).all()
    if kind == "negative":   # the force formula has no such case
        return
    inside = 8 * math.sqrt(2) if dtype == torch.float64 else 6 * math.sqrt(2)
    rho = ((q > inside ** 2) & (q < (inside + 1.5) ** 2)).to(dtype)
    F = hgh_local_grad(nuc, [p], g, rho)[0]
    for c in range(3):
        want, size = float((rho * dV[c]).sum()) * g.dV, float((rho * dV[c]).abs().sum()) * g.dV
        if math.isnan(want):
            assert math.isnan(float(F[c]))
        else:
            rel = 16 * (1 + (inside + 1.5) ** 2) * eps + 4 * 2.0 ** -53 * g.L * (inside + 1.5) / p.r_loc
            assert abs(float(F[c]) - want) <= rel * size, (c, float(F[c]), want)
