"""Compensated and accurate sums whose splits pass FLT_MAX on the way and come back: the sources'
tiles are summed apart, and 2.5e38 + 2.5e38 - 3.2e38 is 1.8e38.

Tolerance: the terms' own errors (5e-7 of 2.5e38 each, compensated) against the result: 2e-6."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["compensated", "accurate"])
@pytest.mark.parametrize("grads", [False, True])
@pytest.mark.parametrize("nt", [1, 700])
def test_a_sum_that_comes_back(prec, grads, nt):
    import torch

    import omega3d_gb300 as G
    ns = 1024
    x = np.zeros((3, ns), np.float32)
    x[0] = 1.0
    s = np.zeros((3, ns), np.float32)
    s[1, 0], s[1, 256], s[1, 512] = 2.5e38, 2.5e38, -3.2e38
    r = np.full(ns, 1e-3, np.float32)
    t = np.zeros((3, nt), np.float32)
    targ = G.Points(torch.from_numpy(t).cuda(), inert=True)
    G.points_affect_points(G.Points(*(torch.from_numpy(a).cuda() for a in (x, s, r))), targ,
                           G.ResultsType("velandgrad" if grads else "velonly"), G.ExecEnv("rm", prec))
    uo, _ = O.points_affect_points(x, r, s, t, None, True, "rm", 2)
    u = targ.u.cpu().numpy()
    assert np.abs(uo[2]).min() > 1.7e38
    assert (u[:2] == 0).all() and (np.abs(u[2] - uo[2]) <= 2e-6 * np.abs(uo[2])).all()
