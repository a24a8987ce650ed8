"""Transfer Gamma from distinct triple products (many modes) against the permanents of single pairs
(one late and one primordial mode at a time take that route): fewer, exactly and more than the ten
samples of the zero rule, unsorted and repeated triples, and magnitudes on both sides of the rule's
threshold.

Tolerance: both routes sum n_mu xsize <= 1e4 products of three table entries, each rounded three
times: 1e4 2^-52 of the sum of magnitudes, which exceeds the largest entry by less than 40 here: 1e-10
of it would be the worst case, sqrt(1e4) 2^-52 40 = 1e-12 the expected one and the bound asked for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ctx(mg, lmax, P, Pp, xsize, tri, prim, amp):
    q, _, cl = mg.workload(lmax, P)
    xvec, qt = mg.transfer_workload(lmax, Pp, xsize)
    c = mg.Context(0)
    c.set_basis(2, lmax, q)
    c.set_modes(tri)
    c.set_spectrum(cl)
    c.set_transfer(xvec, qt * amp, prim)
    return c


@pytest.mark.parametrize("lmax,P,Pp,xsize,amp", [(40, 6, 3, 5, 1.0), (40, 6, 3, 10, 1.0), (61, 5, 4, 11, 1.0), (60, 8, 5, 24, 1.0),
                                                 (40, 6, 3, 9, 1e-11), (40, 6, 3, 14, 3e-12), (40, 6, 3, 14, 1e-13)])
def test_transfer_routes_agree(mg, lmax, P, Pp, xsize, amp):
    rng = np.random.default_rng(xsize)
    tri = rng.integers(0, P, size=(70, 3)).astype(np.int32)
    prim = rng.integers(0, Pp, size=(40, 3)).astype(np.int32)
    with _ctx(mg, lmax, P, Pp, xsize, tri, prim, amp) as c:
        G = c.gamma_transfer(0.7)
    scale = np.abs(G).max()
    for m, n in rng.integers(0, 40, size=(25, 2)):
        with _ctx(mg, lmax, P, Pp, xsize, tri[m:m + 1], prim[n:n + 1], amp) as c:
            g = c.gamma_transfer(0.7)[0, 0]
        assert abs(G[m, n] - g) <= 1e-12 * scale, (m, n)
