"""One pair at a time against the FP64 oracle where the packed FP32 cores change form: the
edges of the Gaussian polynomial's intervals and its far-field limit, the smallest and largest
separations, coincident points and zero radii.

Tolerances, relative per target, from the operations' rounding bounds (2^-24 each, hardware
reciprocal square root 2^-22): the longest chain is the Gaussian gradient factor, 2.5 times
the error of q plus 5 times that of 1/sigma plus the polynomial's 1.8e-7; below 5e-6 plain
and, with the corrected reciprocal square root, below 2e-6 compensated."""
import numpy as np
import pytest

import oracle as O
from omega3d_gb300.metrics import rel_err

pytestmark = pytest.mark.gpu

TOL = {"plain": 5e-6, "compensated": 2e-6}


def _q_values():
    edges = np.arange(0.0, 49.0)
    q = [0.0, 1e-12, 1e-6, 0.5, 46.999, 47.5, 48.0, 49.0, 100.0, 1e4, 1e8]
    for e in edges[1:]:
        q += [e * (1 - 3e-7), e, e * (1 + 3e-7)]
    return np.array(q)


@pytest.mark.parametrize("prec", ["plain", "compensated"])
@pytest.mark.parametrize("core", ["gauss", "rm", "wl", "v2"])
@pytest.mark.parametrize("sr,tr", [(0.02, 0.015), (0.02, None), (3.0, 0.001), (0.0, None)])
def test_one_pair_at_the_core_edges(core, prec, sr, tr):
    import torch

    import omega3d_gb300 as G
    assert torch.cuda.is_available()
    q = _q_values()
    sig = np.sqrt(np.float32(sr) ** 2 + (0.0 if tr is None else np.float32(tr) ** 2))
    if sr == 0.0:
        q, sig = q[q > 0], 0.02          # no core at all: singular at every distance
    rng = np.random.default_rng(5)
    q = rng.permutation(np.tile(q, 3))
    d = rng.normal(size=(3, q.size))
    d *= np.sqrt(q) * sig / np.linalg.norm(d, axis=0)
    x = np.zeros((3, 1), np.float32)
    s = np.array([[0.3], [-0.7], [1.1]], np.float32)
    r = np.full(1, sr, np.float32)
    t = d.astype(np.float32)
    rt = None if tr is None else np.full(q.size, tr, np.float32)

    def dev(a):
        return torch.from_numpy(a).to("cuda")

    targ = G.Points(dev(t), None, None if rt is None else dev(rt), inert=rt is None)
    G.points_affect_points(G.Points(dev(x), dev(s), dev(r)), targ, G.ResultsType("velandgrad"), G.ExecEnv(core, prec))
    uo, go = O.points_affect_points(x, r, s, t, rt, True, core, 2)
    keep = np.ones(q.size, bool)
    if sr == 0.0:
        # closer than 2.8e-8 with no core, the WL gradient factor's parts (5 d^-5) pass FLT_MAX
        keep = 5.0 / np.linalg.norm(t.astype(np.float64), axis=0) ** 5 < np.finfo(np.float32).max
        assert keep.sum() > 0.95 * q.size
    uo, go = uo[:, keep], go[:, keep]
    ug, gg, t = targ.u.cpu().numpy()[:, keep], targ.ug.cpu().numpy()[:, keep], t[:, keep]
    assert np.isfinite(ug).all() and np.isfinite(gg).all()
    # every target against its own magnitude: one term, in which r3 s and b3 d (s x d) add up
    assert rel_err(gg, go, floor=1e-30)[0] <= TOL[prec]
    moving = np.linalg.norm(uo, axis=0) > 0
    # the cross product's own rounding is relative to |d||s|, not to |d x s|
    c = np.linalg.norm(np.cross(s.T, t.T, axis=1), axis=1)
    c /= np.maximum(np.linalg.norm(t, axis=0) * np.linalg.norm(s), 1e-30)
    e = np.linalg.norm(ug - uo, axis=0)[moving] / np.linalg.norm(uo, axis=0)[moving]
    assert (e * np.minimum(c[moving], 1.0)).max() <= TOL[prec]
