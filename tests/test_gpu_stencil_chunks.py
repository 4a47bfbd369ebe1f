"""The plane-marching stencil where its x chunks and edge tiles change: one plane per CTA, uneven last
chunks, rows and columns past the edge, against shifted sums in FP64 torch.

A value is at most fifteen roundings of terms that add up to `size`; its dot with psi a sum of N^3 of them.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def lap(p, order):
    cf = {2: (-6.0, (1.0,)), 4: (-7.5, (16.0 / 12.0, -1.0 / 12.0))}[order]
    out, size = cf[0] * p, abs(cf[0]) * p.abs()
    for ax in (-3, -2, -1):
        n = p.shape[ax]
        for d, c in enumerate(cf[1], start=1):
            for a, b in ((d, 0), (0, d)):
                if n > d:
                    out.narrow(ax, a, n - d).add_(p.narrow(ax, b, n - d), alpha=c)
                    size.narrow(ax, a, n - d).add_(p.narrow(ax, b, n - d).abs(), alpha=abs(c))
    return out, size


@pytest.mark.parametrize("shape", [(1, 2, 4, 4), (1, 16, 16, 16), (3, 17, 33, 36), (1, 40, 40, 40), (4, 64, 64, 64),
                                   (1, 80, 80, 80), (2, 5, 100, 8), (1, 200, 34, 32)])
@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
def test_stencil(shape, order, dtype):
    from gato_gb300.operators import stencil
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    psi = torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda").to(dtype)
    V = torch.randn(*shape[1:], generator=g, dtype=torch.float64, device="cuda").to(dtype)
    h, coef = 0.25, -0.5 / 0.25 ** 2
    out, dot = stencil(psi, h, "dirichlet", order, coef, V=V, dot=True)
    ref, size = lap(psi.double(), order)
    ref, size = coef * ref + V.double() * psi.double(), abs(coef) * size + (V.double() * psi.double()).abs()
    eps = 2.0 ** (-53 if dtype == torch.float64 else -24)
    # FP32 forms differences to the centre: its intermediate terms are up to twice the size
    assert float(((out.double() - ref).abs() / size).max()) < 40 * eps
    want, scale = (ref * psi.double()).flatten(1).sum(1) * h ** 3, (size * psi.double().abs()).flatten(1).sum(1) * h ** 3
    assert float(((dot - want).abs() / scale).max()) < 40 * eps
