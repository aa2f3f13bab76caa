"""The block substitution at the edges of its tiles: orders around the 64-row block and the 16-wide K
chunk, the smallest one, the first whose rows are prefetched (n > 384) and ones whose column block is
16 wide (n > 576), with fewer columns than a tile, a full tile and a remainder.  LAPACK's test ratio (xGET02: ||b - A x||_1 / (||A||_1 ||x||_1 eps)
< 30) per column, on random well-conditioned matrices whose rows are shuffled so that the
factorisation pivots."""
import numpy as np
import pytest

import rayleigh_b200 as rb

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.mark.parametrize("n", [2, 14, 16, 18, 62, 64, 66, 128, 130, 194, 384, 386, 450, 578, 898])
@pytest.mark.parametrize("ncols", [1, 16, 32, 39])
def test_substitution_edges(n, ncols):
    rng = np.random.Generator(np.random.PCG64(n * 100 + ncols))
    count = 3
    a = rng.standard_normal((count, n, n)) / np.sqrt(n) + 2.0 * np.eye(n)
    a = np.stack([m[rng.permutation(n)] for m in a])          # [matrix][row][col]
    cm = np.ascontiguousarray(a.transpose(0, 2, 1))           # column-major per matrix
    b = rng.standard_normal((count, ncols, n))
    with rb.BatchedLU(n, count) as lu:
        lu.factor(cm)
        x, _, _ = lu.solve(b)
    r = b - np.matmul(x, cm)
    an = np.abs(cm).sum(axis=2).max(axis=1)
    ratio = np.abs(r).sum(axis=2) / (an[:, None] * np.abs(x).sum(axis=2) * EPS)
    assert ratio.max() < 30.0, float(ratio.max())


def test_factors_from_memory_take_about_as_long_as_from_cache():
    """One column for 8 and for 64 systems of order 768: both are a single wave with a CTA an SM, so that
    the one difference is that the factors of 64 (302 MB) come from HBM on every call and those of 8
    (38 MB) stay in L2.  Rows that are not on their way early enough show as a ratio of 1.6; with the
    prefetches it is 1.25."""
    n = 768
    rng = np.random.Generator(np.random.PCG64(768))
    a = rng.standard_normal((n, n)) / np.sqrt(n) + 2.0 * np.eye(n)
    ms = {}
    for count in (8, 64):
        b = rng.standard_normal((count, 1, n))
        with rb.BatchedLU(n, count) as lu:
            lu.factor(np.repeat(a[None], count, 0))
            ms[count] = min(lu.solve(b)[2] for _ in range(20))
    print(ms)
    assert ms[64] < 1.42 * ms[8], ms
