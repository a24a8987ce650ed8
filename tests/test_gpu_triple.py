"""FP64 Gamma by distinct triple products (full mode lists) and by permanents (few modes of a large
basis), against the permanents of the downloaded M table in numpy: pair counts below, at and just
past the 32 x 64 tiles, node counts below and past one chunk of 16, split and unsplit sums, unsorted
and repeated triples, node ranges.

Tolerance.  Both sides sum n_mu <= 500 products of three entries, each rounded three times:
(n_mu + 3) 2^-53 of the sum of magnitudes at most, 6e-14; the magnitudes exceed the largest Gamma by
less than 2 for these lists, so 2e-13 of the largest entry."""
import numpy as np
import pytest
from conftest import rel_max

pytestmark = pytest.mark.gpu
PERMS = ((0, 1, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0), (1, 0, 2), (0, 2, 1))


def _reference(c, tri, k0=0, k1=None):
    M = c.get_mij()
    _, w = c.get_gl()
    k1 = w.size if k1 is None else k1
    M, w = M[:, :, k0:k1], w[k0:k1] / (48 * np.pi)
    N = len(tri)
    G = np.zeros((N, N))
    for m in range(N):
        for s in PERMS:
            G[m] += (M[tri[m, 0], tri[:, s[0]]] * M[tri[m, 1], tri[:, s[1]]] * M[tri[m, 2], tri[:, s[2]]]) @ w
    return G


def _ctx(mg, lmax, P, tri):
    q, _, _ = mg.workload(lmax, P)
    c = mg.Context(0)
    c.set_basis(2, lmax, q)
    c.set_modes(tri)
    c.init_glint()
    return c


# P = 1, 2: one partial tile; 7: U = 28; 10: U = 55, UV = 1540; 11: U = 66 (past two u tiles)
@pytest.mark.parametrize("lmax,P,N", [(4, 1, 1), (9, 2, 4), (12, 7, 84), (60, 10, 220), (330, 11, 286), (40, 20, 3), (40, 24, 1)])
def test_gamma_fp64_routes(mg, lmax, P, N):
    rng = np.random.default_rng(P)
    tri = rng.integers(0, P, size=(N, 3)).astype(np.int32)  # unsorted, with repeats
    with _ctx(mg, lmax, P, tri) as c:
        G = c.gamma(mg.PREC_FP64)
        ref = _reference(c, tri)
        n = c.get_gl()[0].size
        parts = c.gamma_partial(mg.PREC_FP64, 0, 1) + c.gamma_partial(mg.PREC_FP64, 1, n)
    assert np.array_equal(G, G.T)
    assert rel_max(G, ref) <= 2e-13
    assert rel_max(parts, ref) <= 2e-13
