"""Force integrals on the FP64 grids whose coordinate tables come to 48 KB (N = 2038 .. 2048): the tables share
that with the kernels' own arrays, so the launch has to opt in to more.

The density is zero outside one small block, over which the integral is restated in plain torch. Bound, in
eps of the sum of the terms' magnitudes: 512 for the order of the 512 terms, 8 for a term's evaluation, and
1900 for the coordinates (either side to 2 eps of L / 2 = 10.2; a term changes by at most 46 of itself per bohr).
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2040, 2048])
def test_forces(N):
    from gato_gb300.geometry import Nuclei
    from gato_gb300.grid import Grid3D
    from gato_gb300.potentials import multi_center_softened_coulomb_grad
    from gato_gb300.pseudopotentials import hgh_local_grad, lookup
    if torch.cuda.mem_get_info()[0] < 90e9:
        pytest.skip("needs a 69 GB density")
    h = 0.01
    grid = Grid3D(N, N * h)
    nuc = Nuclei(torch.tensor([[0.4, -0.3, 0.2]], dtype=torch.float64), torch.tensor([1.0], dtype=torch.float64))
    rho = torch.zeros(N, N, N, dtype=torch.float64, device="cuda")
    o, b = N // 2 + 3, 8
    block = torch.rand(b, b, b, generator=torch.Generator().manual_seed(N), dtype=torch.float64)
    rho[o:o + b, o:o + b, o:o + b] = block.cuda()
    x = -N * h / 2 + (torch.arange(o, o + b, dtype=torch.float64) + 0.5) * h
    d = torch.stack(torch.meshgrid(x - 0.4, x + 0.3, x - 0.2, indexing="ij"))
    eps = 0.05
    w = -block / ((d ** 2).sum(0) + eps ** 2) ** 1.5
    p = lookup("H")
    r = d.norm(dim=0).requires_grad_()
    u = r / p.r_loc
    v = -p.Z_ion / r * torch.erf(u / 2 ** 0.5) + torch.exp(-u ** 2 / 2) * sum(c * u ** (2 * i) for i, c in enumerate(p.c))
    (dv,) = torch.autograd.grad(v.sum(), r)
    for got, f in ((multi_center_softened_coulomb_grad(nuc, grid, rho, eps), w * d),
                   (hgh_local_grad(nuc, [p], grid, rho), -block * dv / r.detach() * d)):
        want = f.sum((1, 2, 3)) * h ** 3
        bound = (512 + 8 + 1900) * 2.0 ** -52 * f.abs().sum((1, 2, 3)) * h ** 3
        assert ((got.cpu().reshape(3) - want).abs() < bound).all()
    del rho
    torch.cuda.empty_cache()
