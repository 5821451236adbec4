"""GPU test of the triangular solves at the edges of their blocks.

One solve with the factors and no refinement after it (the loop stops at a relative residual of
0.5).  The matrix is 4 I plus a random part of spectral norm 2, so its condition number is below 4.
The factorisation's trailing updates round their operands to TF32 (2^-12 on average): entries of L
near 1 / (4 sqrt n) times entries of U near 1 / sqrt n, n of them, leave an error matrix of norm near
2 sqrt(2) 2^-12 / 4 = 1.7e-4, a relative residual near 4e-5.  Bounded here by 2e-4; a wrong or missing
block would leave 1e-2 or more.
"""

import numpy as np
import pytest

import omega3d_gb300 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 511, 512, 513, 641, 1024, 1100, 1700])
@pytest.mark.parametrize("K", [1, 2, 3, 8])
def test_one_solve_without_refinement(n, K):
    rng = np.random.default_rng(n + K)
    A = (rng.normal(size=(n, n)) / np.sqrt(n) + 4.0 * np.eye(n)).astype(np.float32)
    A = A[rng.permutation(n)]   # the pivots are off the diagonal
    b = rng.normal(size=(K, n)).astype(np.float32)
    bem = G.BEM(n)
    bem.set_block(0, 0, np.ascontiguousarray(A.T))
    bem.factor()
    if K == 1:
        _, x = bem.solve(b[0], tol=0.5, max_iter=1, x64=True)
        x = x[None]
    else:
        _, x = bem.solve_many(b, tol=0.5, max_iter=1, x64=True)
    r = b.astype(np.float64) - x @ A.astype(np.float64).T
    assert (np.linalg.norm(r, axis=1) <= 2e-4 * np.linalg.norm(b, axis=1)).all()
