"""GPU test of the close panel pairs of the influence matrix where a warp takes 2 to 32 of the listed pairs
(one where the list has fewer than the launch has warps).  Tolerance and reference as the other
coefficient tests': 1e-5 of an entry plus 1e-6 of the largest, against the oracle in double."""

import numpy as np
import pytest

import omega3d_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,maxlev", [(80, 3), (130, 2), (200, 2), (320, 2), (320, 1)])
def test_lists_around_the_number_of_warps(m, maxlev):
    import torch
    nodes, idx = G.generate_ovoid(2, 2.0, 2.0, 2.0)
    nodes, idx = np.asarray(nodes, np.float32), np.asarray(idx).reshape(-1, 3)[:m]
    s = G.Surfaces(nodes, idx.ravel().copy(), nunk=2)
    t = G.Surfaces(nodes * np.float32(1.2), idx.ravel().copy(), nunk=2)
    out = torch.full((2 * m, 2 * m), float("nan"), device="cuda")
    G.panels_on_panels_coeff(s.device_arrays("cuda"), t.device_arrays("cuda"), 2, False, out, maxlev=maxlev)
    c = out.cpu().numpy()
    geo = [dict(nodes=q.x, idx=q.idx, area=q.area, x1=q.x1, x2=q.x2, norm=q.norm) for q in (s, t)]
    ref = O.panels_on_panels_coeff(geo[0], geo[1], 2, False, "rm", 2, maxlev=maxlev)
    assert np.all(np.abs(c - ref) <= 1e-5 * np.abs(ref) + 1e-6 * np.abs(ref).max())
