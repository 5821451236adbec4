"""The LU factorisation at the edges of its panels, sub-panels, column groups and clusters: sizes
around multiples of 8, 64, 128, 512 and of the rows one block of a cluster holds (640),
matrices that force an interchange at every column, ties, and columns without a usable pivot.

The solution is refined to a relative residual of 1e-10; the check recomputes it in FP64 from
the FP32 matrix and the FP64 solution (numpy), with a bound of 1e-9."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(A, b):
    import torch

    import omega3d_gb300 as G
    n = A.shape[0]
    bem = G.BEM(n)
    bem.set_block(0, 0, torch.from_numpy(np.ascontiguousarray(A.T)).cuda())     # column-major
    _, x = bem.solve(torch.from_numpy(b).cuda(), tol=1e-10, x64=True)
    return x.cpu().numpy(), bem


def _residual(A, x, b):
    return np.linalg.norm(A.astype(np.float64) @ x - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 63, 64, 65, 72, 127, 128, 129, 191, 193, 511, 513, 576, 639, 640, 641,
                               1279, 1281, 2561])
def test_sizes_around_the_panels(n):
    rng = np.random.default_rng(n)
    A = rng.normal(size=(n, n)).astype(np.float32)
    A[np.arange(n), np.arange(n)] += np.float32(2.5 * np.sqrt(n) + 1.0)     # well conditioned
    A = A[rng.permutation(n)]
    b = rng.normal(size=n).astype(np.float32)
    x, _ = _solve(A, b)
    assert _residual(A, x, b) <= 1e-9


@pytest.mark.parametrize("n", [96, 700, 1500])
def test_every_column_interchanges(n):
    # a dominant diagonal moved by a random permutation of the rows: the pivots are anywhere
    rng = np.random.default_rng(n + 1)
    A = (rng.normal(size=(n, n)) / np.sqrt(n)).astype(np.float32)
    A[np.arange(n), np.arange(n)] += np.float32(4.0)
    A = A[rng.permutation(n)]
    b = rng.normal(size=n).astype(np.float32)
    x, _ = _solve(A, b)
    assert _residual(A, x, b) <= 1e-9


@pytest.mark.parametrize("n", [40, 136, 664])
def test_ties(n):
    # blocks of an 8 x 8 Hadamard matrix, rows and columns permuted: eight equal magnitudes in
    # every column, condition number 1
    rng = np.random.default_rng(n + 2)
    h = np.array([[1.0]])
    for _ in range(3):
        h = np.block([[h, h], [h, -h]])
    A = np.kron(np.eye(n // 8), h)[rng.permutation(n)][:, rng.permutation(n)].astype(np.float32)
    b = rng.normal(size=n).astype(np.float32)
    x, _ = _solve(A, b)
    assert _residual(A, x, b) <= 1e-9
    y, _ = _solve(A, b)
    assert np.array_equal(x, y)     # the same pivots every time


@pytest.mark.parametrize("what", ["zero", "nan"])
@pytest.mark.parametrize("n,col", [(64, 0), (200, 63), (700, 130), (1300, 1299)])
def test_column_without_a_pivot_is_reported(n, col, what):
    import omega3d_gb300 as G
    rng = np.random.default_rng(3)
    A = rng.normal(size=(n, n)).astype(np.float32)
    A[:, col] = 0.0 if what == "zero" else np.nan
    with pytest.raises(G.O3GError, match="singular|SINGULAR|pivot|converge"):
        _solve(A, np.ones(n, np.float32))
    # and the next system is solved
    A = np.eye(n, dtype=np.float32)
    x, _ = _solve(A, np.ones(n, np.float32))
    assert np.array_equal(x, np.ones(n))
