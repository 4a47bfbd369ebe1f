"""Lone real fields on the half-spectrum passes against the generic engine's full complex solves.

A field with no imaginary part (a Hartree density, the one pair of a one-orbital system, the last pair
of an odd count) takes two rows per z line and the N + 1 columns that hold a Hermitian spectrum. Both
sides compute the same sums, so they agree to a few roundings per transform level: 25 levels of three
axes there and back, a factor of four for their accumulation, gives 100 eps (2e-14 and 1.2e-5 at most;
norms of random errors stay well below).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = {torch.float64: 100 * 2.0 ** -53, torch.float32: 100 * 2.0 ** -24}
# every register shape, the packed ones among them
SIZES = [16, 18, 20, 24, 28, 30, 32, 36, 40, 42, 48, 50, 54, 56, 60, 64, 70, 72, 80, 84, 90, 96, 98, 100, 108, 112,
         120, 126, 128, 140, 144, 160]


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def smooth(n, N, seed, dtype):
    g = torch.Generator().manual_seed(seed)
    a = (torch.arange(N, dtype=torch.float64) + 0.5) / N - 0.5
    X, Y, Z = torch.meshgrid(a, a, a, indexing="ij")
    c = 0.2 * torch.rand(n, 4, generator=g, dtype=torch.float64) - 0.1
    f = torch.stack([torch.exp(-30 * ((X - k[0]) ** 2 + (Y - k[1]) ** 2 + (Z - k[2]) ** 2)) * (1 + k[3] * Z) for k in c])
    f = f * (1 + 0.1 * torch.rand(n, N, N, N, generator=g, dtype=torch.float64))
    return f.to(dtype).cuda().contiguous()


def both(plan, call):
    """call() on the plan's default engine and on the generic one."""
    from gato_gb300.autotune import set_plan
    got = call()
    set_plan(plan, 0, 1)
    ref = call()
    set_plan(plan, 0, 0)
    return got, ref


@pytest.mark.parametrize("N", SIZES)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
def test_hartree(N, dtype):
    from gato_gb300.solvers.poisson import PoissonPlan
    h = 10.0 / N
    plan = PoissonPlan(N, h, h / 2, dtype, 1)
    rho = smooth(1, N, N, dtype)[0]
    got, ref = both(plan, lambda: plan.potential(rho))
    assert rel(got, ref) < TOL[dtype]
    # new contents of the same buffers, smaller by far: nothing of the first solve stays behind
    small = (1e-3 * rho.flip(0)).contiguous()
    got, ref = both(plan, lambda: plan.potential(small))
    assert rel(got, ref) < TOL[dtype]


@pytest.mark.parametrize("N", SIZES)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
def test_every_shape_solves_pairs(N, dtype):
    """Two fields of two pair densities (the multi-field z forward) on every register shape."""
    from gato_gb300.solvers.poisson import PoissonPlan
    h = 10.0 / N
    plan = PoissonPlan(N, h, h / 2, dtype, 2)
    orb, psi = smooth(4, N, N + 1, dtype), smooth(1, N, 5, dtype)[0]
    got, ref = both(plan, lambda: plan.exchange_into(psi, orb, torch.zeros_like(psi)))
    assert rel(got, ref) < TOL[dtype]


@pytest.mark.parametrize("n", [1, 2, 3])
@pytest.mark.parametrize("N", [24, 40, 50, 64, 96])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
def test_exchange_block_and_energy(N, n, dtype):
    from gato_gb300.grid import Grid3D
    from gato_gb300.scf import Operator, pair_fields
    from gato_gb300.solvers.poisson import PoissonPlan
    h = 10.0 / N
    plan = PoissonPlan(N, h, h / 2, dtype, pair_fields(n))
    orb = smooth(n, N, 7 * N + n, dtype)
    psi = smooth(1, N, 3, dtype)[0]
    got, ref = both(plan, lambda: plan.exchange_into(psi, orb, torch.full_like(psi, 0.5), 0.7))
    assert rel(got - 0.5, ref - 0.5) < 4 * TOL[dtype] * float(ref.norm() / (ref - 0.5).norm())
    op = Operator(Grid3D(N, 10.0), dtype, 4)
    op.set_exchange(plan, orb)
    for epi in (0, 1, 2):
        op.tune(epi)
        got, ref = both(plan, op.apply_block)
        assert rel(got, ref) < TOL[dtype], epi
    got, ref = both(plan, lambda: op.energy_terms(None)[3:].cpu())
    np.testing.assert_allclose(got.numpy(), ref.numpy(), rtol=TOL[dtype])
