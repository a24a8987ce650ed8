"""Householder panels of the eigensolver at row blocks that end inside, at and
beyond the kernel's passes over a CTA's rows (16 and fewer rows, 24 per pass of
the row sums, 32 per pass of the last step), and columns with nothing below the
subdiagonal.  The matrices are D + rank two (two reflections of a diagonal), so
their eigenvalues are D's; bound 8 n eps max|D|, eps = 2^-52."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 17, 18, 31, 33, 49, 400, 2431, 2433, 3648, 3650, 4864, 4866])
def test_known_spectrum(mg, n):
    rng = np.random.default_rng(n)
    d = np.sort(rng.standard_normal(n) * np.exp(rng.uniform(-6, 1, n)))
    A = np.diag(d)
    for _ in range(2):
        u = rng.standard_normal(n)
        u /= np.linalg.norm(u)
        Au = A @ u
        A = A - 2 * np.outer(u, Au) - 2 * np.outer(Au, u) + 4 * (u @ Au) * np.outer(u, u)
    A = (A + A.T) / 2
    c = mg.Context(0)
    try:
        w = c.eigh(A, False)[0]
    finally:
        c.close()
    assert np.max(np.abs(w - d)) <= 8 * max(n, 4) * np.finfo(float).eps * np.max(np.abs(d))


@pytest.mark.parametrize("n", [40, 200])
def test_trivial_reflectors(mg, n):
    A = np.diag(np.arange(1.0, n + 1))
    for k in range(0, n - 1, 3):  # pairs: every third column couples to the next only
        A[k, k + 1] = A[k + 1, k] = 0.5
    c = mg.Context(0)
    try:
        w, V = c.eigh(A, True)
    finally:
        c.close()
    eps = np.finfo(float).eps
    assert np.max(np.abs(w - np.linalg.eigvalsh(A))) <= 8 * n * eps * n
    assert np.max(np.abs(V @ V.T - np.eye(n))) <= 8 * n * eps
