"""FP64-accurate tensor-core products with every number of slices (digit products run
two groups at a time, the first alone for an odd number), K inside, at and beyond a
block of 512, ragged M and N, and rows whose exponents leave the range in which the
result is scaled by bit patterns.  Bound per element, with scales 2^e < 2 max|.| and digits p at
most 2^-7p: the s - 1 dropped products with p + q = s and the digits cut off both factors make
4 (s + 1) 2^-7s < 2^(6 - 7 s) per term, the sums 2^-48: K (2^-48 + 2^(6 - 7 s)) max|a_m| max|b_n|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(mg):
    c = mg.Context(0)
    yield c
    c.close()


def check(ctx, A, B, s):
    C = ctx.gemm_f64(A, B, slices=s)
    K = A.shape[1]
    with np.errstate(under="ignore"):
        ref = (A.astype(np.longdouble) @ B.astype(np.longdouble))
        bound = K * (2.0 ** -48 + 2.0 ** (6 - 7 * s)) * np.abs(A).max(1)[:, None].astype(np.longdouble) * np.abs(B).max(0)[None, :]
    assert np.all(np.abs(C - ref) <= bound + 5e-324)


@pytest.mark.parametrize("s", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (63, 65, 31), (64, 129, 512), (130, 128, 545), (257, 66, 1090)])
def test_groups(ctx, s, M, N, K):
    rng = np.random.default_rng(M + N + K)
    check(ctx, rng.standard_normal((M, K)), rng.standard_normal((K, N)), s)


def test_extreme_rows(ctx):
    rng = np.random.default_rng(1)
    A, B = rng.standard_normal((40, 70)), rng.standard_normal((70, 50))
    A *= np.exp2(np.linspace(-900, 500, 40))[:, None]
    B *= np.exp2(np.linspace(-500, 400, 50))[None, :]
    A[3] = 0.0
    B[:, 7] = 0.0
    check(ctx, A, B, 8)
