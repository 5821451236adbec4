"""GPU test of the close panel pairs of the influence matrix: every depth of the subdivision, and
numbers of panels around the 32 pairs that one warp takes.  The targets are the sources' panels or the same
ones scaled by 1.2, so that all pairs are close and none of their centroids coincide.  Tolerance: the
panel tests' own, 1e-5 of an entry plus 1e-6 of the largest, against the oracle in double (its float
sums over 4,096 leaves are themselves off by 1.8e-6 of the largest here)."""

import numpy as np
import pytest

import omega3d_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu


def _geo(s):
    return dict(nodes=s.x, idx=s.idx, area=s.area, x1=s.x1, x2=s.x2, norm=s.norm)


@pytest.mark.parametrize("nunk", [2, 3])
@pytest.mark.parametrize("maxlev", [1, 2, 3])
@pytest.mark.parametrize("m", [1, 2, 5, 6, 33])
def test_close_pairs(m, maxlev, nunk):
    import torch
    nodes, idx = G.generate_ovoid(2, 2.0, 2.0, 2.0)
    nodes, idx = np.asarray(nodes, np.float32), np.asarray(idx).reshape(-1, 3)[:m]
    s = G.Surfaces(nodes, idx.ravel().copy(), nunk=nunk)
    t = G.Surfaces(nodes * np.float32(1.2), idx.ravel().copy(), nunk=nunk)
    n = m * nunk
    for targ, is_self in ((s, True), (t, False)):
        out = torch.full((n, n), float("nan"), device="cuda")
        G.panels_on_panels_coeff(s.device_arrays("cuda"), targ.device_arrays("cuda"), nunk, is_self, out, maxlev=maxlev)
        c = out.cpu().numpy()
        ref = O.panels_on_panels_coeff(_geo(s), _geo(targ), nunk, is_self, "rm", 2, maxlev=maxlev)
        assert np.all(np.abs(c - ref) <= 1e-5 * np.abs(ref) + 1e-6 * np.abs(ref).max())
