"""Gauss-Legendre nodes at the sizes where the kernel changes course: one or more recurrences per
root (below about n = 31), the reciprocal chunks of 256 steps, blocks of 32 roots, the middle root
in a block of its own.  Bounds as for the sizes that the library has always been checked at: nodes
5e-16, weights 1e-13 against the long-double oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 5, 8, 9, 16, 17, 29, 30, 32, 62, 63, 64, 65, 127, 255, 256, 257, 513])
def test_gl_nodes_edges(mg, orc, n):
    x, w = mg.gl_nodes(n)
    xo, wo = orc.gl_nodes(n)
    assert np.max(np.abs(x - xo)) <= 5e-16
    assert np.max(np.abs(w - wo) / wo) <= 1e-13
    assert np.array_equal(x, -x[::-1]) and np.array_equal(w, w[::-1])


@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 95, 96, 97])
def test_gl_nodes_chunk_edges(mg, orc, n):
    """The recurrence works in chunks of 32 steps: a first step past a whole chunk, and one short of it."""
    test_gl_nodes_edges(mg, orc, n)
