"""The FP64 correction sweep on basis entries that are subnormal in FP32, as the tails of decaying vectors are:
W = 0.8 v_2 + 1.1 r + 0.5 v_0 loses its v_0 part there too.

The products run in FP32, where such an entry has the spacing 2^-149: one rounding an entry, one a product sum,
for three vectors 6 * 2^-149, and 8 eps of the FP64 values.
"""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2000, 2001])
@pytest.mark.parametrize("tail", [2.0 ** -128, 2.0 ** -140, 2.0 ** -148])
def test_tails(n, tail):
    from gato_gb300 import _lib
    j, m, cut = 2, 4, n // 2
    g = torch.Generator(device="cuda").manual_seed(n)
    Q = torch.zeros(4, n, dtype=torch.float64, device="cuda")
    Q[:, :cut] = torch.linalg.qr(torch.randn(cut, 4, generator=g, dtype=torch.float64, device="cuda"))[0].T
    Q[:, cut:] = tail * (1 + torch.rand(4, n - cut, generator=g, dtype=torch.float64, device="cuda"))
    K = torch.zeros(m + 1, n, dtype=torch.float64, device="cuda")
    K[: j + 1] = Q[: j + 1]
    K[j + 1] = 0.8 * Q[2] + 1.1 * Q[3] + 0.5 * Q[0]
    a, b = torch.zeros(m, dtype=torch.float64, device="cuda"), torch.zeros(m, dtype=torch.float64, device="cuda")
    _lib.call("gato_lanczos_step", _lib.F64, n, 1.0, C.c_void_p(K.data_ptr()), j, m, 1, 1, C.c_void_p(a.data_ptr()),
              C.c_void_p(b.data_ptr()), C.c_void_p(_lib.stream()))
    got, want = K[j + 1, cut:] * b[j], 1.1 * Q[3, cut:]
    assert float((got - want).abs().max()) < 6 * 2.0 ** -149 + 8 * 2.0 ** -53 * float(want.abs().max())
