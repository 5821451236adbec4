"""The LU factorisation at the numbers of rows where its panels change kernels: one block of 256, 512
or 640 rows and one more, 16 blocks of 256, 512 and 640 and one more (10,241: no cluster).

The solution is refined to a relative residual of 1e-10; the check recomputes it in FP64, with a bound of
1e-9.  A factorisation that was wrong somewhere would not converge."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 257, 512, 514, 640, 642, 4096, 4097, 8192, 8193, 10240, 10241])
def test_rows_at_the_kernels_edges(n):
    import torch

    import omega3d_gb300 as G
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, n, device="cuda", generator=g) / n ** 0.5
    A += 4.0 * torch.eye(n, device="cuda")
    A = A[torch.randperm(n, device="cuda", generator=g)]          # the pivots are anywhere
    b = torch.randn(n, device="cuda", generator=g)
    bem = G.BEM(n)
    bem.set_block(0, 0, A.t().contiguous())                       # column-major
    _, x = bem.solve(b, tol=1e-10, x64=True)
    r = A.double() @ x - b.double()
    assert bem.iters <= 5
    assert float(r.norm() / b.double().norm()) <= 1e-9
