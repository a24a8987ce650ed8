"""Adjoint routes at their edges against torch float64 autograd (tests/adjoint_torch.py): pair counts
below and past one 32-row tile, one and several splits, one basis function, few modes of a large
basis (cofactors per pair instead of triple products), unsorted and repeated triples, shapes of one
and of five terms.  Bound: 1e-11 relative, as for the sizes always checked (both sides sum about
1e3 products, each rounded a few times, into gradients of mixed sign)."""
import adjoint_torch as at
import numpy as np
import pytest
import torch
from conftest import rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,P,N,terms", [(6, 1, 1, 1), (30, 3, 10, 5), (64, 7, 84, 1), (65, 8, 100, 2), (40, 20, 3, 1)])
def test_vjp_routes(mg, lmax, P, N, terms):
    rng = np.random.default_rng(100 + P)
    tri = rng.integers(0, P, size=(N, 3)).astype(np.int32)
    q, _, cl = mg.workload(lmax, P)
    shapes = mg.separable_shapes(lmax, 3, 21, terms, terms)
    with mg.Context(0) as c:
        c.set_basis(2, lmax, q)
        c.set_modes(tri)
        c.set_spectrum(cl)
        c.init_glint()
        mu, w = c.get_gl()
        up, upb = rng.standard_normal((N, N)), rng.standard_normal((3, N))
        dg, db = c.gamma_vjp(up), c.project_gl_vjp(shapes, upb)
        beta, _ = c.project_gl(shapes)
    pr = at.Problem(mu, w, 2, lmax, tri, cl, shapes)
    qt = torch.tensor(q, requires_grad=True)
    (pr.gamma(qt) * torch.tensor(up)).sum().backward()
    assert rel_fro(dg, qt.grad.numpy()) <= 1e-11
    qt = torch.tensor(q, requires_grad=True)
    b_ref, _ = pr.beta_norm2(qt)
    assert rel_fro(beta, b_ref.detach().numpy()) <= 1e-12
    (b_ref * torch.tensor(upb)).sum().backward()
    assert rel_fro(db, qt.grad.numpy()) <= 1e-11


@pytest.mark.parametrize("P,N", [(2, 4), (6, 1)])
def test_vjps_of_one_node(mg, P, N):
    """A quadrature of the single node 0, antisymmetric like a Gauss-Legendre rule; both routes of each."""
    rng = np.random.default_rng(P)
    q, _, cl = mg.workload(7, P)
    tri = rng.integers(0, P, size=(N, 3)).astype(np.int32)
    shapes = mg.separable_shapes(7, 2, 23, 1, 2)
    mu, w = np.zeros(1), np.full(1, 2.0)
    up, upb = rng.standard_normal((N, N)), rng.standard_normal((2, N))
    with mg.Context(0) as c:
        c.set_basis(2, 7, q)
        c.set_modes(tri)
        c.set_spectrum(cl)
        c.set_gl(mu, w)
        dg, db = c.gamma_vjp(up), c.project_gl_vjp(shapes, upb)
    pr = at.Problem(mu, w, 2, 7, tri, cl, shapes)
    for got, loss in ((dg, lambda t: (pr.gamma(t) * torch.tensor(up)).sum()),
                      (db, lambda t: (pr.beta_norm2(t)[0] * torch.tensor(upb)).sum())):
        qt = torch.tensor(q, requires_grad=True)
        loss(qt).backward()
        assert rel_fro(got, qt.grad.numpy()) <= 1e-11


@pytest.mark.parametrize("lmax,P,N,S", [(40, 2, 4, 15), (40, 4, 20, 20), (40, 4, 2, 20), (87, 3, 10, 12), (170, 5, 35, 16)])
def test_projection_vjp_of_many_and_few_modes(mg, lmax, P, N, S):
    """Shape tensors where the modes are many for the basis (all but the third case), cofactors else."""
    rng = np.random.default_rng(7 + P)
    tri = mg.mode_triples(P)[:N]
    q, _, cl = mg.workload(lmax, P)
    shapes = mg.separable_shapes(lmax, S, 25, 2, 2)
    upb = rng.standard_normal((S, N))
    with mg.Context(0) as c:
        c.set_basis(2, lmax, q)
        c.set_modes(tri)
        c.set_spectrum(cl)
        c.init_glint()
        mu, w = c.get_gl()
        db = c.project_gl_vjp(shapes, upb)
    qt = torch.tensor(q, requires_grad=True)
    (at.Problem(mu, w, 2, lmax, tri, cl, shapes).beta_norm2(qt)[0] * torch.tensor(upb)).sum().backward()
    assert rel_fro(db, qt.grad.numpy()) <= 1e-11
