"""The accurate mode's pair term to its last bits: two sources whose terms cancel to 2^-25 of each, so
that the float result shows the terms' errors of 2^-44.

Bound on the rms error over 1,000 such pairs, in units of 2^-44 of a term, from the rounding steps of
one term (each uniform, rms its bound over sqrt 3): the squared distance 8 steps of 0.05, the root's
residual 3 of 0.19, its correction 2 of 0.1, the low parts 3 of 0.125: 0.25, and 0.36 for two terms.  The
square of the residual left out adds up to 15/8 2^-44 to each term."""
import decimal

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_cancelling_pairs():
    import torch

    import omega3d_gb300 as G
    D = decimal.Decimal
    rng = np.random.default_rng(4)
    sr = np.float32(0.1)
    r = torch.full((2,), float(sr), device="cuda")
    env = G.ExecEnv("rm", "accurate")
    err = []
    with decimal.localcontext() as ctx:
        ctx.prec = 50
        s2 = D(float(sr)) ** 2
        for _ in range(1000):
            d1, d2, w1 = (np.float32(v) for v in (*rng.uniform(0.5, 4.0, 2), rng.uniform(1.0, 2.0)))

            def term(d, w):
                return D(float(d)) * D(float(w)) / (D(float(d)) ** 2 + s2).sqrt() ** 3

            a1 = term(d1, w1)
            w2 = np.float32(float(a1 / term(d2, 1.0)))
            x = torch.tensor([[-d1, d2], [0, 0], [0, 0]], dtype=torch.float32, device="cuda")
            s = torch.tensor([[0, 0], [w1, w2], [0, 0]], dtype=torch.float32, device="cuda")
            t = G.Points(torch.zeros(3, 1, device="cuda"), inert=True, grads=False)
            G.points_affect_points(G.Points(x, s, r), t, G.ResultsType("velonly"), env)
            err.append(float((D(float(t.u[2, 0])) + a1 - term(d2, w2)) / a1))
    assert np.sqrt(np.mean(np.square(err))) <= 0.36 * 2.0 ** -44
