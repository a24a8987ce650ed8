"""The single-precision projection kernel at the edges of its tiling, against
the FP64 projection of the same shapes: row blocks of 128 rows per parity (the
second block opens at l_max = 258), chunks of 32 lattice points, operand widths
of 16, 32, 48 and 64 basis columns, passes of four terms, one shape per item and
partly filled items.

Tolerance.  Each shape value carries about ten FP32 roundings of 2^-24, its
product with the basis is exact to 2^-24, and the sums over rows and slabs round
at 2^-24 of partial sums that exceed the result by a modest factor (the
oscillating basis): 1e-6 relative per shape for P <= 32 and 2e-6 beyond, the
bounds the FP32 form has always been held to."""
import numpy as np
import pytest
from conftest import rel_fro

pytestmark = pytest.mark.gpu


def _ctx(mg, lmin, lmax, P):
    cl = mg.synthetic_cl(lmax)
    c = mg.Context(0)
    c.set_basis(lmin, lmax, mg.weighted_q(mg.legendre_q(lmin, lmax, P), cl, lmin))
    c.set_modes(mg.mode_triples(P))
    c.set_spectrum(cl)
    return c


@pytest.mark.parametrize("lmin,lmax,P,terms,S", [
    (2, 3, 2, 1, 1), (2, 17, 3, 4, 2), (5, 64, 16, 5, 3), (2, 257, 17, 1, 1), (2, 258, 16, 4, 5), (3, 259, 8, 8, 2),
    (2, 300, 33, 2, 3), (2, 130, 48, 3, 2), (2, 131, 49, 1, 9), (2, 90, 64, 4, 1), (2, 515, 4, 2, 4)])
def test_f32_projection_edges(mg, lmin, lmax, P, terms, S):
    shapes = mg.separable_shapes(lmax, S, seed=7, tmin=terms, tmax=terms) + mg.bump_shapes(2, seed=8)
    with _ctx(mg, lmin, lmax, P) as c:
        b64 = c.project(shapes, mg.PREC_FP64)
        b32 = c.project(shapes, mg.PREC_SPLIT)
        again = c.project(shapes, mg.PREC_SPLIT)
        batch = c.project_batch(shapes, mg.PREC_SPLIT)
    assert np.array_equal(b32, again) and np.array_equal(b32, batch)
    for s in range(len(shapes)):
        assert rel_fro(b32[s], b64[s]) <= (1e-6 if P <= 32 else 2e-6), (s, rel_fro(b32[s], b64[s]))


def test_f32_projection_ignores_table_entries_below_lmin(mg):
    """l < l_min takes no part: infinities and NaN there (a power law at l = 0) leave the result alone."""
    lmax = 60
    shapes = mg.separable_shapes(lmax, 3, seed=9, tmin=1, tmax=3)
    dirty = [dict(s, tab=s["tab"].copy()) for s in shapes]
    for s in dirty:
        s["tab"][:, :, 0] = np.inf
        s["tab"][:, :, 1] = np.nan
    with _ctx(mg, 2, lmax, 5) as c:
        clean = c.project(shapes, mg.PREC_SPLIT)
        got = c.project(dirty, mg.PREC_SPLIT)
    assert np.array_equal(got, clean)


def test_f32_batch_replays_after_another_range(mg):
    """The captured batch uses the slab schedule of its own range: a projection at another l_max in
    between makes it plan again."""
    q1, tr, cl = mg.workload(150, 6)
    q2, _, cl2 = mg.workload(90, 6)
    shapes = mg.config_shapes(150, ("mix", 6, 1, 2), seed=3)
    with _ctx(mg, 2, 150, 6) as c:
        first = c.project_batch(shapes, mg.PREC_SPLIT)
        c.set_basis(2, 90, q2)
        c.set_spectrum(cl2)
        c.project(mg.config_shapes(90, ("mix", 6, 1, 2), seed=4), mg.PREC_SPLIT)
        c.set_basis(2, 150, q1)
        c.set_spectrum(cl)
        assert np.array_equal(c.project_batch(shapes, mg.PREC_SPLIT), first)


@pytest.mark.parametrize("lmax,small", [(200, 5e-22), (2000, 5e-20)])
def test_f32_projection_of_a_small_spectrum(mg, lmax, small):
    """C_l + N_l in units where products of three point-weight factors (2l+1)^{5/6} / sqrt(C_l) exceed
    the FP32 range although the weights do not: within the form's 1e-6."""
    cl = mg.synthetic_cl(lmax)
    cl *= small / cl[2:].min()
    shapes = mg.separable_shapes(lmax, 3, seed=11, tmin=1, tmax=2) + mg.bump_shapes(1, seed=12)
    for s in shapes[:3]:
        s["tab"][:, 0] *= 1e-12  # keeps the sums over points in range
    with mg.Context(0) as c:
        c.set_basis(2, lmax, mg.legendre_q(2, lmax, 6))
        c.set_modes(mg.mode_triples(6))
        c.set_spectrum(cl)
        b64 = c.project(shapes[:3], mg.PREC_FP64)
        b32 = c.project(shapes[:3], mg.PREC_SPLIT)
    for s in range(3):
        assert rel_fro(b32[s], b64[s]) <= 1e-6, (s, rel_fro(b32[s], b64[s]))


@pytest.mark.parametrize("P", [2, 16, 33])
@pytest.mark.parametrize("l", [3, 5])
def test_f32_projection_of_one_odd_multipole(mg, P, l):
    """l_min = l_max odd has no points (i + j + k is odd): its beta is zero whatever the context
    computed before."""
    with _ctx(mg, 2, 64, P) as c:
        c.project(mg.bump_shapes(9, seed=14), mg.PREC_SPLIT)
        c.set_basis(l, l, np.random.default_rng(P).standard_normal((1, P)))
        c.set_spectrum(mg.synthetic_cl(l))
        shapes = mg.bump_shapes(9, seed=15)
        b64 = c.project(shapes, mg.PREC_FP64)
        b32 = c.project(shapes, mg.PREC_SPLIT)
    assert not b64.any() and not b32.any()


def test_f32_projection_of_a_shape_that_overflows_outside_the_triangle(mg):
    """f(i) g(j) h(k) = 1e45 at points with k > i + j, which no sum contains, and 0 at those that count."""
    lmax = 60
    shape = mg.separable_shapes(lmax, 1, seed=13, tmin=2, tmax=2)[0]
    l = np.arange(lmax + 1)
    shape["tab"][0] = [np.where(l <= 3, 1e15, 0.0), np.where(l <= 3, 1e15, 0.0), np.where(l >= 12, 1e15, 0.0)]
    with _ctx(mg, 2, lmax, 5) as c:
        b64 = c.project([shape], mg.PREC_FP64)
        b32 = c.project([shape], mg.PREC_SPLIT)
        tame = dict(shape, tab=shape["tab"] * [[[1e-12]], [[1.0]]])  # bounded: the same values at the points that count
        batch = [c.project_batch([x], mg.PREC_SPLIT) for x in (tame, shape, tame)]
    assert rel_fro(b32, b64) <= 1e-6
    assert np.array_equal(batch[1], b32) and np.array_equal(batch[0], batch[2])
    assert rel_fro(batch[0], b64) <= 1e-6


@pytest.mark.parametrize("c,sigma", [((1e17, -2e17, 5e16), 1e17), ((3e16, 0.3, 0.7), 0.1), ((0.21, 0.3141, 0.4759), 1e-21),
                                     ((0.2, 0.3, 0.5), 1e30), ((1e40, 0.0, 0.0), 1e40)])
def test_f32_projection_of_extreme_bumps(mg, c, sigma):
    """Centres and widths far from 1 are numbers like any other: a constant, or zero everywhere."""
    shape = [{"kind": mg.SHAPE_BUMP, "c": np.array(c), "sigma": sigma}]
    with _ctx(mg, 2, 60, 5) as ctx:
        b64 = ctx.project(shape, mg.PREC_FP64)
        b32 = ctx.project(shape, mg.PREC_SPLIT)
    assert np.all(np.isfinite(b64))
    assert np.linalg.norm(b32 - b64) <= 1e-6 * np.linalg.norm(b64)


def test_f32_projection_long_row_sums_keep_small_addends(mg):
    """Nine terms at l_max = 2000, three passes of up to 17 accumulators per row (past the 32 that are added
    plainly): in the slab j = 1000 the point k = j outweighs each later block of 32 points by more than 2^24,
    their sum not.  Tolerance: the roundings of a point (weight, shape, product), of the fold and of the slab
    sum, 2^-24 each at most, several of them averaged over 500 rows: 1.5e-7."""
    lmax = 2000
    tab = np.zeros((9, 3, lmax + 1))
    tab[0] = 1.0
    tab[0, :, 1000] = 3 * 2.0**30
    with mg.Context(0) as c:
        c.set_basis(2, lmax, np.ones((lmax - 1, 1)))
        c.set_modes(np.zeros((1, 3), np.int32))
        c.set_spectrum(np.ones(lmax + 1))
        shape = [{"kind": mg.SHAPE_SEPARABLE, "tab": tab}]
        b64 = c.project(shape, mg.PREC_FP64)
        b32 = c.project(shape, mg.PREC_SPLIT)
    assert rel_fro(b32, b64) <= 1.5e-7


@pytest.mark.parametrize("P", [30, 33])
def test_f32_projection_fold_keeps_small_addends(mg, P):
    """Every slab's first row, l = 2, outweighs each other one by 2^24 or more.  Tolerance: rows are added in
    groups of 16 before the compensated sum, 15 additions that round by half a unit, 2^-25, at most."""
    lmax = 1000
    tab = np.ones((1, 3, lmax + 1))
    tab[:, 0, 2] = 3 * 2.0**30
    with mg.Context(0) as c:
        c.set_basis(2, lmax, mg.legendre_q(2, lmax, P))
        c.set_modes(np.zeros((1, 3), np.int32))
        c.set_spectrum(np.ones(lmax + 1))
        shape = [{"kind": mg.SHAPE_SEPARABLE, "tab": tab}]
        b64 = c.project(shape, mg.PREC_FP64)
        b32 = c.project(shape, mg.PREC_SPLIT)
    assert rel_fro(b32, b64) <= 15 * 2.0**-25


@pytest.mark.parametrize("P", [30, 33])
def test_f32_projection_fold_keeps_small_addends(mg, P):
    """Every slab's first row, l = 2, outweighs each other one by 2^24 or more.  Tolerance: rows are added in
    groups of 16 before the compensated sum, 15 additions that round by half a unit, 2^-25, at most."""
    lmax = 1000
    tab = np.ones((1, 3, lmax + 1))
    tab[:, 0, 2] = 3 * 2.0**30
    with mg.Context(0) as c:
        c.set_basis(2, lmax, mg.legendre_q(2, lmax, P))
        c.set_modes(np.zeros((1, 3), np.int32))
        c.set_spectrum(np.ones(lmax + 1))
        shape = [{"kind": mg.SHAPE_SEPARABLE, "tab": tab}]
        b64 = c.project(shape, mg.PREC_FP64)
        b32 = c.project(shape, mg.PREC_SPLIT)
    assert rel_fro(b32, b64) <= 15 * 2.0**-25


@pytest.mark.parametrize("P", [5, 20, 40, 60])
@pytest.mark.parametrize("terms", [36, 40, 48, 60])
def test_f32_projection_sum_modes(mg, terms, P):
    """The four ways of the sums, by the number of roundings that the terms' passes add at l_max = 130: plain,
    groups of 16 rows compensated, groups of 8, everything compensated; for each operand width, and again with a
    term that overflows outside the triangle (masked and compensated)."""
    lmax = 130
    shapes = mg.separable_shapes(lmax, 2, seed=16, tmin=terms, tmax=terms) + mg.bump_shapes(1, seed=17)
    l = np.arange(lmax + 1)
    far = [dict(s, tab=s["tab"].copy()) for s in shapes[:2]] + shapes[2:]
    for s in far[:2]:
        s["tab"][0] = [np.where(l <= 3, 1e15, 0.0), np.where(l <= 3, 1e15, 0.0), np.where(l >= 12, 1e15, 0.0)]
    with _ctx(mg, 2, lmax, P) as c:
        for sh in (shapes, far):
            b64 = c.project(sh, mg.PREC_FP64)
            b32 = c.project(sh, mg.PREC_SPLIT)
            assert np.array_equal(b32, c.project_batch(sh, mg.PREC_SPLIT))
            for s in range(3):
                assert rel_fro(b32[s], b64[s]) <= (1e-6 if P <= 32 else 2e-6), (s, rel_fro(b32[s], b64[s]))
