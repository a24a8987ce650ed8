"""Single-precision projection of narrow bumps whose coefficients cancel most: every shape
within the form's 1e-6 of the FP64 projection (relative 2-norm), at the benchmark's size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,P", [(500, 20), (2000, 30)])
def test_cancelling_bumps(mg, lmax, P):
    q, tr, cl = mg.workload(lmax, P)
    bumps = mg.bump_shapes(128, seed=1)
    shapes = [bumps[i] for i in (14, 30, 63, 65, 78, 105, 123)]
    with mg.Context(0) as c:
        c.set_basis(2, lmax, q)
        c.set_modes(tr)
        c.set_spectrum(cl)
        b64 = c.project(shapes, mg.PREC_FP64)
        b32 = c.project(shapes, mg.PREC_SPLIT)
    err = np.linalg.norm(b32 - b64, axis=1) / np.linalg.norm(b64, axis=1)
    assert np.all(err <= 1e-6), err
