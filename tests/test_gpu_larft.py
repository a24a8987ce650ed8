"""The block reflectors' triangular factors, built by rows (modal_eigh's
back-transformation): sizes on both sides of one and two blocks of 256
reflectors and of a warp's rows, and matrices with trivial reflectors (tau = 0)
inside a block.  Bounds of a backward stable solver, with eps = 2^-52:
||A V^T - V^T diag(w)||_F <= 8 n eps ||A|| max(1, sqrt(n)/4), |V V^T - I| <= 8 n eps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["dense", "split"])
@pytest.mark.parametrize("n", [4, 6, 34, 37, 255, 257, 258, 261, 511, 513, 514, 769])
def test_reflector_blocks(mg, n, kind):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    A = A + A.T
    if kind == "split":  # decoupled blocks: columns with nothing below the subdiagonal
        for cut in (n // 3, n // 2):
            A[cut:, :cut] = 0.0
            A[:cut, cut:] = 0.0
    c = mg.Context(0)
    try:
        w, V = c.eigh(A, True)
    finally:
        c.close()
    eps = np.finfo(float).eps
    tol = 8 * n * eps
    assert np.linalg.norm(A @ V.T - V.T * w[None, :]) <= tol * np.max(np.abs(w)) * max(1.0, np.sqrt(n) / 4)
    assert np.max(np.abs(V @ V.T - np.eye(n))) <= tol
