"""One pair at a time in the accurate mode against the FP64 oracle, where its double-single core changes
form: the edges of the Gaussian polynomial's intervals, q near 0 (where 2 q - 1 rounds), its far-field
limit, and separations from far below to far above the radii.

Tolerances, relative per target: the velocity's term carries about 41 bits (the polynomial 8.8e-11,
the neglected square of the root's residual 2^-41, the cross product 2^-46 of |d||s|), so what
remains is the output's rounding, 6e-8 of each component: 1e-7.  A gradient is the sum of two float terms of
at most six roundings each: 1e-6."""

import numpy as np
import pytest

import oracle as O
from omega3d_gb300.metrics import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("core", ["gauss", "rm"])
@pytest.mark.parametrize("sr,tr", [(0.02, 0.015), (0.02, None), (3.0, 0.001)])
def test_one_pair(core, sr, tr):
    import torch

    import omega3d_gb300 as G
    q = [0.0, 1e-12, 1e-8, 1e-6, 1e-3, 0.25, 0.4999999, 0.5, 0.5000001, 47.5, 48.0, 49.0, 100.0, 1e4, 1e8]
    for e in range(1, 49):
        q += [e * (1 - 3e-7), float(e), e * (1 + 3e-7)]
    rng = np.random.default_rng(7)
    q = rng.permutation(np.tile(q, 3))
    sig = np.sqrt(np.float32(sr) ** 2 + (0.0 if tr is None else np.float32(tr) ** 2))
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
    G.points_affect_points(G.Points(dev(x), dev(s), dev(r)), targ, G.ResultsType("velandgrad"),
                           G.ExecEnv(core, "accurate"))
    uo, go = O.points_affect_points(x, r, s, t, rt, True, core, 2)
    ug, gg = targ.u.cpu().numpy(), targ.ug.cpu().numpy()
    assert np.isfinite(ug).all() and np.isfinite(gg).all()
    assert rel_err(gg, go, floor=1e-30)[0] <= 1e-6
    # (nearly parallel to the strength the cross product's own rounding counts)
    sine = np.linalg.norm(np.cross(s.T, t.T, axis=1), axis=1)
    sine = sine / np.maximum(np.linalg.norm(t.astype(np.float64), axis=0) * np.linalg.norm(s), 1e-300)
    keep = sine > 1e-3
    assert keep.sum() > 0.9 * (q > 0).sum()
    assert (np.linalg.norm(ug - uo, axis=0)[keep] <= 1e-7 * np.linalg.norm(uo, axis=0)[keep]).all()
