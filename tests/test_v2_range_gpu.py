"""The V2 core where d^4 leaves FP32's range: separations above 4.3e9, where it overflows and the
term is 0 (the true one is below 1e-19 of the strength), and below 5.6e-12 with no core, where it
underflows and the plain term is infinite.  One such pair must not spoil the others' sums: a parked
particle without strength, and the padding of the source tiles at (1e9, 1e9, 1e9) against a far target.

Tolerances as the other pair tests': 5e-6 plain, 2e-6 compensated, of the FP64 oracle's term."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

TOL = {"plain": 5e-6, "compensated": 2e-6}


def _run(x, s, r, t, prec, entry):
    import torch

    import omega3d_gb300 as G
    X, S, R, T = (torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda() for a in (x, s, r, t))
    if entry == "points":
        targ = G.Points(T, inert=True)
        G.points_affect_points(G.Points(X, S, R), targ, G.ResultsType("velandgrad"), G.ExecEnv("v2", prec))
        return targ.u.cpu().numpy(), targ.ug.cpu().numpy()
    z = [torch.zeros(k, n, device="cuda") for n in (X.shape[1], T.shape[1]) for k in (3, 9)]
    G.Batch([G.BatchSystem(X, S, R, z[0], z[1], T, z[2], z[3])], G.ExecEnv("v2", prec)).run()
    torch.cuda.synchronize()
    return z[2].cpu().numpy(), z[3].cpu().numpy()


def _check(x, s, r, t, prec, entry, grads=True):
    u, g = _run(x, s, r, t, prec, entry)
    a = [np.ascontiguousarray(v, np.float32) for v in (x, r, s, t)]
    uo, go = O.points_affect_points(*a, None, True, "v2", 2)
    assert np.isfinite(g).all()
    for got, ref in ((u, uo),) + (((g, go),) if grads else ()):
        assert np.isfinite(got).all()
        assert (np.linalg.norm(got - ref, axis=0) <= TOL[prec] * np.linalg.norm(ref, axis=0)).all()


@pytest.mark.parametrize("entry", ["points", "batch"])
@pytest.mark.parametrize("prec", ["plain", "compensated"])
class TestFar:
    def test_parked_particle(self, prec, entry):
        _check([[0.0, 1e10], [0.0, -2e10], [0.0, 3e12]], [[1.0, 0.0], [2.0, 0.0], [3.5, 0.0]], [0.1, 0.1],
               [[1.0, 0.3], [2.0, -0.1], [3.0, 0.2]], prec, entry)

    def test_padding_against_a_far_target(self, prec, entry):
        # 3e9 from the source (d^4 near 8e37; the gradient's d^-5 is below FP32's range) and more than 4.3e9
        # from the padding
        _check([[0.0], [0.0], [0.0]], [[1.0], [2.0], [-3.0]], [0.1],
               [[-2.0e9, -3.0e9], [-1.5e9, -1.0e8], [-1.7e9, -2.0e8]], prec, entry, grads=False)

    def test_a_pair_out_of_range_is_zero(self, prec, entry):
        t = np.array([[5e9, 1e10, 1e12, 1e15], [0.0, 1.0, 1e12, 0.0], [0.0, 0.0, -1e11, 3e14]])
        u, g = _run(np.zeros((3, 1)), [[1.0], [2.0], [3.0]], [0.1], t, prec, entry)
        assert (u == 0).all() and (g == 0).all()


@pytest.mark.parametrize("entry", ["points", "batch"])
def test_no_core_and_a_vanishing_separation(entry):
    # d^4 is 0: (d x s) r3 is infinite where d x s is not 0, as with the root taken exactly
    u, _ = _run(np.zeros((3, 1)), [[1.0], [2.0], [0.0]], [0.0], [[1e-12, 1.0], [1e-12, 0.0], [1e-12, 0.0]], "plain",
                entry)
    assert np.isinf(u[:, 0]).all() and np.isfinite(u[:, 1]).all()
