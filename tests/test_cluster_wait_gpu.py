"""The bounded waits of the LU panels that run in one thread-block cluster: o3g_debug_wait_test(2) makes each of
them poll a phase that nothing completes, for a short time.  The factorisation gives up with
O3G_ERR_TIMEOUT, and the next one and its solve succeed, for each of the three block sizes, with one
block and with a whole cluster."""
import pytest

import omega3d_gb300 as G
from omega3d_gb300 import _lib as L

pytestmark = pytest.mark.gpu

TIMEOUT = 6


@pytest.mark.parametrize("n", [5, 200, 1000, 4096, 4200, 9000])
def test_exchanges_run_out_and_the_next_factorisation_succeeds(n, cuda):
    import torch
    lib = L.lib()
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, n, generator=g, device="cuda") / n ** 0.5
    A.diagonal().add_(3.0)
    b = torch.randn(n, generator=g, device="cuda")
    bem = G.BEM(n)
    bem.set_block(0, 0, A.t().contiguous())
    torch.cuda.synchronize()
    assert lib.o3g_debug_wait_test(2) == 0
    try:
        st = lib.o3g_bem_factor(bem.h, None)
    finally:
        assert lib.o3g_debug_wait_test(0) == 0
    assert st == TIMEOUT, lib.o3g_last_error().decode()
    assert "timed out" in lib.o3g_last_error().decode()
    bem.factor()
    _, x = bem.solve(b, tol=1e-10, max_iter=30, x64=True)
    r = b.double() - A.double() @ x
    assert bem.relres <= 1e-10 and float(r.norm() / b.double().norm()) <= 1e-9
