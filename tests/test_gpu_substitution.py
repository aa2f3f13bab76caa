"""The block substitution at the edges of its tiles: orders around the 64-row block and the 16-wide K
chunk, the smallest one and one whose column block is 16 wide (n > 576), with fewer columns than a
tile, a full tile and a remainder.  LAPACK's test ratio (xGET02: ||b - A x||_1 / (||A||_1 ||x||_1 eps)
< 30) per column, on random well-conditioned matrices whose rows are shuffled so that the
factorisation pivots."""
import numpy as np
import pytest

import rayleigh_b200 as rb

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.mark.parametrize("n", [2, 14, 16, 18, 62, 64, 66, 128, 130, 194, 578])
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
