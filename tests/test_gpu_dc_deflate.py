"""Divide and conquer where much deflates: whole merges, runs of negligible couplings between
entries that do not, repeated eigenvalues (rotations in a row), and ties in the final order.
Bounds of the eigensolver's other tests (eps = 2^-52): eigenvalues 8 n eps ||A||, residual the
same times max(1, sqrt(n) / 4), orthogonality 8 n eps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def matrix(kind, n, rng):
    if kind == "identity plus rank one":
        u = rng.standard_normal(n)
        return np.eye(n) + np.outer(u, u) / n
    if kind == "repeated":
        Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
        d = np.repeat(rng.standard_normal((n + 6) // 7), 7)[:n]
        A = (Q * d) @ Q.T
        return (A + A.T) / 2
    if kind == "weakly coupled":  # tridiagonal, most couplings far below rounding
        A = np.diag(np.round(rng.uniform(0, 4, n)))
        e = np.where(rng.uniform(size=n - 1) < 0.2, 0.3, 1e-18)
        return A + np.diag(e, 1) + np.diag(e, -1)
    A = np.diag(np.abs(np.arange(n) - (n - 1) / 2))  # Wilkinson: close pairs
    return A + np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1)


@pytest.mark.parametrize("kind", ["identity plus rank one", "repeated", "weakly coupled", "wilkinson"])
@pytest.mark.parametrize("n", [2, 3, 31, 64, 257, 600])
def test_deflation(mg, n, kind):
    A = matrix(kind, n, np.random.default_rng(n))
    c = mg.Context(0)
    try:
        w, V = c.eigh(A, True)
    finally:
        c.close()
    eps, nrm = np.finfo(float).eps, np.max(np.abs(np.linalg.eigvalsh(A)))
    tol = 8 * max(n, 4) * eps
    assert np.all(np.diff(w) >= 0)
    assert np.max(np.abs(w - np.linalg.eigvalsh(A))) <= tol * nrm
    assert np.linalg.norm(A @ V.T - V.T * w[None, :]) <= tol * nrm * max(1.0, np.sqrt(n) / 4)
    assert np.max(np.abs(V @ V.T - np.eye(n))) <= tol
