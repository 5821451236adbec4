"""The multipliers of the LU panels are IEEE quotients.  2 x 2 blocks [[p, 0], [x, 1]] with right-hand
side (1, 0) and no refinement give -x / p exactly as the factorisation rounded it.  Quotients as close
as they come to the middle between two floats: x / p = (t -+ 1 / p) / 2^25 with t odd, t p = +-1 mod 2^25."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hard_quotients(count, rng):
    ps, xs = [], []
    while len(ps) < count:
        p = int(rng.integers(2 ** 22, 2 ** 23)) * 2 + 1
        inv = pow(p, -1, 2 ** 25)
        for t, e in ((inv, 1), (2 ** 25 - inv, -1)):
            if t > 2 ** 24:
                ps.append(p)
                xs.append((t * p - e) >> 25)
    return np.array(ps[:count], np.float32), np.array(xs[:count], np.float32)


@pytest.mark.parametrize("n,scale", [(64, 1.0), (600, 1.0), (1200, 2.0 ** -70), (4400, 2.0 ** 80)])
def test_quotients(n, scale):
    import omega3d_gb300 as G
    p, x = _hard_quotients(n // 2, np.random.default_rng(n))
    q = -(x / p)
    p, x = p * np.float32(scale), x * np.float32(scale)
    A = np.zeros((n, n), np.float32)
    i = np.arange(0, n, 2)
    A[i, i], A[i + 1, i], A[i + 1, i + 1] = p, x, 1.0
    b = np.zeros(n, np.float32)
    b[::2] = 1.0
    bem = G.BEM(n)
    bem.set_block(0, 0, np.ascontiguousarray(A.T))
    _, got = bem.solve(b, tol=0.5, max_iter=1, x64=True)
    assert np.array_equal(got[1::2].astype(np.float32), q)
