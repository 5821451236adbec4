"""Gradients of planar data: sources and targets in the plane z = 0 with strengths along z, so that every
term of w_z = sum b3 dz c_z is an exact zero (dz = 0), and so must the sums be in every precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _disc(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(3, n)).astype(np.float32)
    x[2] = 0.0
    s = np.zeros((3, n), np.float32)
    s[2] = rng.normal(size=n)
    return x, s


@pytest.mark.parametrize("prec", ["plain", "compensated"])
@pytest.mark.parametrize("core", ["rm", "wl", "exp", "gauss", "v2"])
def test_points(core, prec):
    import torch

    import omega3d_gb300 as G
    x, s = _disc(1500, 1)
    p = G.Points(*(torch.from_numpy(a).cuda() for a in (x, s, np.full(1500, 0.05, np.float32))))
    G.points_affect_points(p, p, G.ResultsType("velandgrad"), G.ExecEnv(core, prec))
    g = p.ug.cpu().numpy()
    assert np.abs(g[0]).max() > 1.0 and np.isfinite(g).all()
    assert (g[8] == 0).all()


@pytest.mark.parametrize("prec", ["plain", "compensated"])
def test_panels(prec):
    import torch

    import omega3d_gb300 as G
    # upright triangles whose centroids lie in the plane: (-h - h + 2 h) / 3 is exact
    c, s = _disc(200, 2)
    h = np.float32(0.01)
    nodes = np.repeat(c, 3, axis=1).reshape(3, 200, 3)
    nodes[0] += h * np.array([-1, 1, 0], np.float32)
    nodes[2] += h * np.array([-1, -1, 2], np.float32)
    surf = G.Surfaces(nodes.reshape(3, 600), np.arange(600, dtype=np.uint32), nunk=2)
    a = surf.device_arrays("cuda")
    a["ts"] = torch.from_numpy(s).cuda()
    t = G.Points(torch.from_numpy(_disc(500, 3)[0]).cuda(), inert=True)
    G.panels_affect_points(surf, t, G.ResultsType("velandgrad"), G.ExecEnv("rm", prec), maxlev=0, arrays=a)
    g = t.ug.cpu().numpy()
    assert np.abs(g[0]).max() > 1.0 and np.isfinite(g).all()
    assert (g[8] == 0).all()
