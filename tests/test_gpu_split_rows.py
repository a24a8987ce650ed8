"""Split Gamma where the sliced rows end inside and beyond what a thread keeps
(K = 3072 nodes after padding to 64) and for few nodes, against the plain FP64
Gamma: 7 digits of 7 bits leave 2^-49 of the row scales, as in the other split
tests 1e-12 of the norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,P", [(2, 1), (21, 2), (42, 3), (85, 5), (2046, 3), (2048, 4), (2091, 3)])
def test_split_rows(mg, lmax, P):
    q, tr, cl = mg.workload(lmax, P)
    with mg.Context(0) as c:
        c.set_basis(2, lmax, q)
        c.set_modes(tr)
        c.init_glint()
        g = c.gamma(mg.PREC_SPLIT).copy()
        ref = c.gamma(mg.PREC_FP64)
    assert np.linalg.norm(g - ref) <= 1e-12 * np.linalg.norm(ref)
