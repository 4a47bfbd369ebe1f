"""One Lanczos step (gato_lanczos_step) against NumPy: shares of the vector per warp, coefficient sums in
groups of eight vectors, alpha and beta summed by their consumers.

With an orthonormal basis and W = F v_j = beta v_{j-1} + alpha v_j + r, r orthogonal to the basis to
rounding (as a Lanczos step meets it), the outputs are alpha, |r| and r / |r|. Sums of n products round like
sqrt(n) eps of their size and W has the basis vectors' size: 300 eps bound every output.
"""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# n: fewer elements than warps, ragged and several shares a warp, an odd n (8-byte loads); j + 1 vectors on
# both sides of a group of eight
@pytest.mark.parametrize("n", [64, 1000, 13824, 262144, 500000, 2001])
@pytest.mark.parametrize("j", [0, 1, 6, 7, 8, 23])
@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
def test_step(n, j, passes, dtype):
    check(n, j, passes, dtype, 0.37)


# basis entries around 1e42 and 1e-42, beyond the FP32 range that the correction's products run in
@pytest.mark.parametrize("dV", [1e-84, 1e84])
@pytest.mark.parametrize("n", [2000, 2001])
def test_step_beyond_fp32_range(n, dV):
    check(n, 5, 1, torch.float64, dV)


def check(n, j, passes, dtype, dV):
    from gato_gb300 import _lib
    m = j + 2
    g = torch.Generator(device="cuda").manual_seed(n + j)
    Q = torch.linalg.qr(torch.randn(n, j + 2, generator=g, dtype=torch.float64, device="cuda"))[0].T / dV ** 0.5
    K = torch.zeros(m + 1, n, dtype=dtype, device="cuda")
    K[: j + 1] = Q[: j + 1].to(dtype)
    W = 0.8 * Q[j] + 1.1 * Q[j + 1] + (0.3 * Q[j - 1] if j > 0 else 0.0)
    K[j + 1] = W.to(dtype)
    a = torch.zeros(m, dtype=torch.float64, device="cuda")
    b = torch.full((m,), 0.3, dtype=torch.float64, device="cuda")
    _lib.call("gato_lanczos_step", _lib.dtype_code(dtype), n, dV, C.c_void_p(K.data_ptr()), j, m, 1, passes,
              C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()), C.c_void_p(_lib.stream()))
    eps = 2.0 ** (-53 if dtype == torch.float64 else -24)
    assert abs(float(a[j]) - 0.8) < 300 * eps
    assert abs(float(b[j]) - 1.1) < 300 * eps
    got, want = K[j + 1].double().cpu().numpy(), Q[j + 1].cpu().numpy()
    assert np.linalg.norm(got - want) * dV ** 0.5 < 300 * eps
