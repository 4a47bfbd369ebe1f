"""The device tridiagonal eigensolver against numpy.linalg.eigh, through gato_lanczos_finish.

The basis is the first m unit vectors of R^n, so the Ritz vectors are the eigenvectors of T themselves.
Eigenvalues come from Sturm counts to the last bit of their bracket: a few eps of the norm of T. An
eigenvector is checked by its residual |T y - lambda y|, a backward-stable solver's few eps of the norm
times the length's growth, by orthogonality where the eigenvalues are apart, and by its sign.
"""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def solve(alpha, beta, K):
    from gato_gb300 import _lib
    m, n = len(alpha), max(256, len(alpha))
    V = torch.zeros(m + 1, n, dtype=torch.float64, device="cuda")
    V[torch.arange(m), torch.arange(m)] = 1.0
    a, b = torch.tensor(alpha, device="cuda"), torch.tensor(beta, device="cuda")
    ev = torch.empty(K, dtype=torch.float64, device="cuda")
    X = torch.empty(K, n, dtype=torch.float64, device="cuda")
    flag = torch.empty(1, dtype=torch.int32, device="cuda")
    P = lambda t: C.c_void_p(t.data_ptr())   # noqa: E731
    _lib.call("gato_lanczos_finish", _lib.F64, n, P(V), m, K, 1e-10, P(a), P(b), P(ev), P(X), P(flag),
              C.c_void_p(_lib.stream()))
    return ev.cpu().numpy(), X.cpu().numpy()[:, :m], int(flag.item())


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 31, 32, 33, 80, 127, 130, 200, 500])
@pytest.mark.parametrize("kind", ["random", "scaled", "huge", "decoupled"])
def test_against_eigh(m, kind):
    rng = np.random.default_rng(m)
    alpha, beta = rng.uniform(-3, 200, m), rng.uniform(0.1, 60, m)
    if kind == "scaled":     # rescaling of the Sturm sequence in both directions
        alpha, beta = alpha * 1e-12, beta * 1e-12
    if kind == "huge":       # beyond 2^100: the exponent is looked at every step
        alpha, beta = alpha * 1e33, beta * 1e33
    if kind == "decoupled":  # exact zeros off the diagonal and repeated eigenvalues
        beta[::3] = 0.0
        alpha[: m // 2] = alpha[0]
    T = np.diag(alpha) + np.diag(beta[: m - 1], 1) + np.diag(beta[: m - 1], -1)
    K = min(m, 6)
    ev, Y, flag = solve(alpha, beta, K)
    lam = np.linalg.eigvalsh(T)
    norm = np.abs(T).sum(1).max()
    assert np.abs(ev - lam[:K]).max() < 16 * EPS * norm
    assert flag == int((beta[: max(m - 1, 1)] < 1e-10).any())
    for k in range(K):
        y = Y[k]
        assert abs(np.linalg.norm(y) - 1) < 64 * EPS
        assert np.linalg.norm(T @ y - ev[k] * y) < 64 * m * EPS * norm
        assert y[np.argmax(np.abs(y))] > 0
    if kind != "decoupled":
        apart = np.abs(lam[:K, None] - lam[None, :K]) > 1e-6 * norm
        G = np.abs(Y @ Y.T) * apart
        assert G.max() < 1e-8
