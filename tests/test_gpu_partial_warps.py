"""FP64 energies on the register shapes whose blocks are not whole warps (M = 40, 56, 60, 84, 180: 80, 112,
120, 196 and 216 threads), against the generic engine: the spectral energy pass and, on a plan too small
for it, the z inverse's energy epilogue. The reductions may exchange only among lanes that exist.

Both engines compute the same sums: 25 levels of three axes there and back, a factor of four for their
accumulation, gives 100 eps.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

RTOL = 100 * 2.0 ** -53


def fields(n, N, seed):
    g = torch.Generator().manual_seed(seed)
    return (torch.rand(n, N, N, N, generator=g, dtype=torch.float64) + 0.1).cuda()


@pytest.mark.parametrize("N", [20, 28, 30, 42, 90])
@pytest.mark.parametrize("n,small", [(1, False), (2, False), (3, False), (3, True)])
def test_energies(N, n, small):
    from gato_gb300.autotune import set_plan
    from gato_gb300.grid import Grid3D
    from gato_gb300.scf import Operator, pair_fields
    from gato_gb300.solvers.poisson import PoissonPlan
    h = 10.0 / N
    plan = PoissonPlan(N, h, h / 2, torch.float64, 1 if small else pair_fields(n))
    orb = fields(n, N, 10 * N + n)
    op = Operator(Grid3D(N, 10.0), torch.float64, 4)
    op.set_exchange(plan, orb)
    rho = (orb ** 2).sum(0).contiguous()
    got = [op.energy_terms(None)[3:].cpu().numpy(), plan.energy(rho).cpu().numpy()]
    set_plan(plan, 0, 1)
    ref = [op.energy_terms(None)[3:].cpu().numpy(), plan.energy(rho).cpu().numpy()]
    for a, b in zip(got, ref):
        np.testing.assert_allclose(a, b, rtol=RTOL)
