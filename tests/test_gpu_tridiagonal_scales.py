"""The device tridiagonal eigensolver at norms far below 1 and with the zero rows that a Lanczos breakdown
leaves: the Sturm sequence shrinks by the norm, or by the distance of a bracket from an eigenvalue 0, each row.

Bounds as in test_gpu_tridiagonal.py, relative to the norm. An eigenvalue that is exactly zero is bracketed to
2^-200 of the norm (twice that, for the bracket's middle).
"""
import numpy as np
import pytest
import torch  # noqa: F401

from test_gpu_tridiagonal import EPS, solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [5, 33, 80, 200])
@pytest.mark.parametrize("scale", [1.0, 1e-17, 1e-45, 2.0 ** -200])
@pytest.mark.parametrize("zeros", [0, 1, 0.5])
def test_scales_and_zero_rows(m, scale, zeros):
    rng = np.random.default_rng(m)
    alpha, beta = rng.uniform(1, 200, m) * scale, rng.uniform(0.1, 0.4, m) * scale   # diagonally dominant: positive
    z = int(zeros * m) if zeros == 0.5 else zeros
    if z:
        alpha[m - z:] = 0.0
        beta[m - z - 1:] = 0.0
    T = np.diag(alpha) + np.diag(beta[: m - 1], 1) + np.diag(beta[: m - 1], -1)
    K = min(m, 6)
    ev, Y, flag = solve(alpha, beta, K)
    unit = np.linalg.eigvalsh(T / scale) * scale
    norm = np.abs(T).sum(1).max()
    assert np.abs(ev - unit[:K]).max() < 16 * EPS * norm
    assert np.abs(ev[:min(z, K)]).max(initial=0.0) <= 2.0 ** -199 * norm
    for k in range(K):
        assert abs(np.linalg.norm(Y[k]) - 1) < 64 * EPS
        assert np.linalg.norm(T / scale @ Y[k] - ev[k] / scale * Y[k]) < 64 * m * EPS * norm / scale
