"""Kernels chained by programmatic dependent launch: a Lanczos run, whose steps chain through every kernel
of both forms, gives the same bits alone, back to back with other runs and beside them on another stream;
sums of many partials match the same energies on the generic engine.

The runs repeat the same kernels on the same inputs, so the comparison is exact. The energies are sums of
the same terms, 25 levels of transform there and back and a factor of four for their accumulation: 100 eps.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def hamiltonian(N, dtype, seed):
    from gato_gb300.grid import Grid3D
    from gato_gb300.hamiltonian import Hamiltonian
    g = torch.Generator().manual_seed(seed)
    V = -torch.rand(N, N, N, generator=g, dtype=torch.float64)
    H = Hamiltonian(Grid3D(N, 0.3 * N), V.to(dtype).cuda(), order=2)
    return H, torch.rand(N, N, N, generator=g, dtype=torch.float64).to(dtype).cuda()


@pytest.mark.parametrize("N,m", [(10, 8), (16, 40), (33, 24), (64, 40), (96, 12)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
def test_lanczos_alone_and_beside_others(N, m, dtype):
    from gato_gb300.solvers.lanczos import lanczos
    sets = [hamiltonian(N, dtype, s) for s in (1, 2)]

    def run(k):
        r = lanczos(sets[k][0], sets[k][1], n_iters=m, n_eigenstates=2)
        return [x for x in (r if isinstance(r, (tuple, list)) else vars(r).values()) if torch.is_tensor(x)]
    want = []
    for k in range(2):
        want.append(run(k))
        torch.cuda.synchronize()
    assert want[0] and all(torch.isfinite(x).all() for x in want[0] if x.is_floating_point())
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = []
    for rep in range(4):
        for k in range(2):
            with torch.cuda.stream(streams[(k + rep) % 2]):
                got.append((k, run(k)))
        got += [(k, run(k)) for k in (1, 0)]
    torch.cuda.synchronize()
    for k, g in got:
        assert all(torch.equal(a, b) for a, b in zip(g, want[k]))


@pytest.mark.parametrize("N,n", [(64, 1), (64, 2), (64, 3), (100, 4)])
def test_energies_of_many_partials(N, n):
    from gato_gb300.autotune import set_plan
    from gato_gb300.grid import Grid3D
    from gato_gb300.scf import Operator, pair_fields
    from gato_gb300.solvers.poisson import PoissonPlan
    g = torch.Generator().manual_seed(N + n)
    orb = torch.rand(n, N, N, N, generator=g, dtype=torch.float64).cuda()
    plan = PoissonPlan(N, 0.2, 0.1, torch.float64, pair_fields(n))
    op = Operator(Grid3D(N, 0.2 * N), torch.float64, 4)
    op.set_exchange(plan, orb)
    got = op.energy_terms(None)[3:].cpu()
    set_plan(plan, 0, 1)
    ref = op.energy_terms(None)[3:].cpu()
    assert float(((got - ref) / ref).abs().max()) < 100 * 2.0 ** -53


@pytest.mark.parametrize("N", [18, 40, 64])
@pytest.mark.parametrize("element", ["O", "Cl", "Li"])   # small boxes, middle ones, boxes as large as the grid
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
def test_projectors_beside_the_stencil(N, element, dtype):
    """A chain of applies, each on the result of the one before, against the same applies one at a time, exactly;
    and one apply against its two parts by themselves, which add the stencil's value and two atoms' projectors in
    another order, at most four roundings of either part's size (a point's sum has ten projectors' terms at most,
    formed alike on both sides)."""
    from gato_gb300.grid import Grid3D
    from gato_gb300.geometry import Nuclei
    from gato_gb300.pseudopotentials import HGH_TABLE, HGHNonlocal
    from gato_gb300.scf import Operator
    g = torch.Generator().manual_seed(N)
    grid = Grid3D(N, 9.0)
    nl = HGHNonlocal(Nuclei(torch.tensor([[0.1, -0.2, 0.3], [0.5, 0.4, -0.6]], dtype=torch.float64),
                            torch.tensor([6.0, 6.0], dtype=torch.float64)), [HGH_TABLE[element]] * 2, grid, dtype)
    psi = torch.rand(N, N, N, generator=g, dtype=torch.float64).to(dtype).cuda()
    op, bare = Operator(grid, dtype, 4), Operator(grid, dtype, 4)
    for o in (op, bare):
        o.set_potential(-psi)
    op.set_nonlocal(nl)
    eps = 2.0 ** -53 if dtype == torch.float64 else 2.0 ** -24
    both, local, far = op.apply(psi).double(), bare.apply(psi).double(), nl(psi).double()
    assert float((both - local - far).norm()) < 4 * eps * float(local.norm() + far.norm())
    bufs = [psi.clone(), torch.empty_like(psi)]
    want = []
    for k in range(6):
        op.apply(bufs[k % 2], bufs[1 - k % 2])
        torch.cuda.synchronize()
        want.append(bufs[1 - k % 2].clone())
        torch.cuda.synchronize()
    for _ in range(3):
        bufs = [psi.clone(), torch.empty_like(psi)]
        for k in range(6):
            op.apply(bufs[k % 2], bufs[1 - k % 2])
        assert torch.equal(bufs[1], want[4]) and torch.equal(bufs[0], want[5])
