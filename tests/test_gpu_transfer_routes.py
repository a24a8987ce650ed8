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


def test_transfer_routes_drop_the_same_samples(mg):
    """The first sample's weight x^2 moved through the zero rule's threshold in steps of one rounding: both
    routes drop it or both keep it (the other samples are zero)."""
    lmax, P, Pp = 40, 6, 3
    rng = np.random.default_rng(3)
    tri = rng.integers(0, P, size=(70, 3)).astype(np.int32)
    prim = rng.integers(0, Pp, size=(40, 3)).astype(np.int32)
    q, _, cl = mg.workload(lmax, P)
    qt = mg.transfer_workload(lmax, Pp, 4)[1] * 1e-12
    qt[1:] = 0.0

    def context(t, p):
        c = mg.Context(0)
        c.set_basis(2, lmax, q)
        c.set_modes(t)
        c.set_spectrum(cl)
        return c, lambda x0: (c.set_transfer(np.array([x0, 1e30, 2e30, 3e30]), qt, p), c.gamma_transfer(1.0))[1]

    cb, both = context(tri, prim)
    for m, n in [(0, 0), (7, 3), (21, 11), (33, 30), (52, 17), (69, 39)]:
        c1, one = context(tri[m:m + 1], prim[n:n + 1])
        lo, hi = 1e-30, 1e29  # kept, dropped
        assert one(lo)[0, 0] != 0.0 and one(hi)[0, 0] == 0.0
        while hi > np.nextafter(lo, hi):
            mid = np.sqrt(lo * hi) if hi > 2 * lo else 0.5 * (lo + hi)
            lo, hi = (mid, hi) if one(mid)[0, 0] != 0.0 else (lo, mid)
        for k in range(-12, 13):
            x = lo + k * (hi - lo)
            assert (both(x)[m, n] != 0.0) == (one(x)[0, 0] != 0.0), (m, n, k)
        c1.close()
    cb.close()
