"""FP64 projection against the oracle where its slabs, rows and sums end inside a
group: rows in eights, sums over k in fours, the basis product's register tiles
(P = 16 | 17, 32 | 33, 45 | 46), slabs of the final sum in eights, several shapes
per launch.  Both sides sum the same few thousand terms in FP64 in different
orders: 1e-12 of the norm, as in the other projection tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmin,lmax,P", [(2, 2, 1), (2, 4, 2), (3, 9, 3), (2, 17, 7), (4, 35, 16), (2, 37, 17),
                                         (9, 50, 32), (2, 51, 33), (3, 52, 45), (2, 53, 46)])
def test_groups(mg, orc, lmin, lmax, P):
    cl = mg.synthetic_cl(lmax)
    rng = np.random.default_rng(lmax)
    q = rng.standard_normal((lmax - lmin + 1, P))
    tr = mg.mode_triples(P)[:: max(1, P // 4)].copy()
    shapes = mg.separable_shapes(lmax, 2, seed=lmax, tmin=1, tmax=3) + mg.bump_shapes(1, seed=P)
    with mg.Context(0) as c:
        c.set_basis(lmin, lmax, q)
        c.set_modes(tr)
        c.set_spectrum(cl)
        beta = c.project(shapes, mg.PREC_FP64)
    for s, sh in enumerate(shapes):
        ref = orc.project(lmin, lmax, q, tr, cl, sh, nthreads=2)
        if lmin == lmax:  # the oracle's walk counts a lone point twice (tetrapyd_count = 2)
            assert orc.tetrapyd_count(lmin, lmax) == 2
            ref = ref / 2
        assert np.linalg.norm(beta[s] - ref) <= 1e-12 * np.linalg.norm(ref), s
