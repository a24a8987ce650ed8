"""l-contractions that fold mirrored quadrature nodes (even and odd l summed apart): odd and even node
counts, odd and even l_min, one l, against the downloaded table's plain sum; nodes that are not
antisymmetric take the unfolded sum.

Tolerance: L <= 200 products of three factors, each rounded three times, summed in either order:
(L + 3) 2^-52 of the sum of magnitudes, 5e-14."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmin,lmax,nmu,P", [(2, 2, 5, 3), (3, 60, 40, 3), (5, 200, 7, 3), (3, 3, 1, 3), (2, 17, 1281, 40),
                                             (3, 16, 1282, 40)])
@pytest.mark.parametrize("shift", [0.0, 1e-6])
def test_m_table_with_and_without_folding(mg, lmin, lmax, nmu, P, shift):
    """(1281 nodes x 820 pairs fill the GPU with full tiles and fold, unless the nodes are shifted.)"""
    x = np.sin(np.pi * (np.arange(nmu) - (nmu - 1) / 2) / (nmu + 1))
    x, w = 0.5 * (x - x[::-1]) + shift, np.ones(nmu)  # exactly antisymmetric for shift = 0
    q = np.random.default_rng(4).standard_normal((lmax - lmin + 1, P))
    with mg.Context(0) as c:
        c.set_basis(lmin, lmax, q)
        c.set_modes(mg.mode_triples(P))
        c.set_gl(x, w)
        c.init_glint()
        M = c.get_mij()
    pl = mg.legendre_table(x, lmax)[:, lmin:]
    ref = np.einsum("kl,lp,lq->pqk", pl, q, q)
    mag = np.einsum("kl,lp,lq->pqk", np.abs(pl), np.abs(q), np.abs(q))
    assert np.all(np.abs(M - ref) <= 5e-14 * mag)
