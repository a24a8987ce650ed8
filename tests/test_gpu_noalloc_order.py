"""The allocation-free FP64 Gamma after smaller calls of the regular path: the
P_l table kernel's shared-memory limit is process-wide, and a small table must
not leave it below what the next caller needs."""
import numpy as np
import pytest
from conftest import rel_max
from test_zz_no_alloc import _call, _regular

pytestmark = pytest.mark.gpu


def test_noalloc_gamma_after_a_smaller_legendre_table(mg):
    torch = pytest.importorskip("torch")
    q, tr, _ = mg.workload(120, 4)
    mg.legendre_table(np.linspace(-1.0, 1.0, 5), 10)
    st, G = _call(mg, torch, q, tr, 2, 120)
    assert st == 0 and rel_max(G, _regular(mg, q, tr, 2, 120)) <= 1e-12
