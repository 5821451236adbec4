"""A graded system that only the narrow triangular solves can take: rows scaled by 1 .. 1e-22 and columns by
1e-22 .. 1 of 2 I + a random part of norm 1/2.  The inverse of its 512 x 512 diagonal block has entries
near 0.003 / (1e-22 1e-22), beyond FLT_MAX; those of its 128 x 128 blocks stay below 1e29.  The
factors are as accurate as for the unscaled matrix (condition below 3), so refinement converges to a
residual of 1e-12, which bounds the scaled solution of the rows scaled by more than 1e-3 to 1e-6 amply."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [512, 640, 1100])
@pytest.mark.parametrize("K", [1, 3])
def test_graded_over_a_block(n, K):
    import omega3d_gb300 as G
    rng = np.random.default_rng(n)
    B = 2.0 * np.eye(n) + rng.normal(size=(n, n)) / (4.0 * np.sqrt(n))
    i = np.minimum(np.arange(n), 511) / 511.0
    d1, d2 = 10.0 ** (-22.0 * i), 10.0 ** (22.0 * (i - 1.0))
    A = np.triu(d1[:, None] * B * d2[None]).astype(np.float32)
    b = (d1 * rng.normal(size=(K, n))).astype(np.float32)
    if K > 1:
        b[1] = 0.0
    bem = G.BEM(n)
    bem.set_block(0, 0, np.ascontiguousarray(A.T))
    if K == 1:
        _, x = bem.solve(b[0], tol=1e-12, max_iter=20, x64=True)
        x = x[None]
        assert bem.relres <= 1e-12
    else:
        _, x = bem.solve_many(b, tol=1e-12, max_iter=20, x64=True)
        assert (bem.relres_many <= 1e-12).all() and (x[1] == 0).all()
    # the same system, unscaled, in FP64 (A's own float entries)
    S = A.astype(np.float64) / d1[:, None] / d2[None]
    xs = np.linalg.solve(S, (b.astype(np.float64) / d1).T).T
    top = d1 > 1e-3   # the rows that the residual's norm sees
    assert np.isfinite(x).all()
    assert np.abs(x * d2 - xs)[:, top].max() <= 1e-6
