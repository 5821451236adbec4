"""The panel kernels' node queues and tile remainders against the oracle: every subdivision
depth, targets so close that nearly every pair subdivides (the queues run full), one to a few
targets, panels or particles more or less than a tile, and field points on the panels.

Tolerance: 1e-5 per target, as every panel test, against the reference's float pair arithmetic
with double sums, in both precisions.  (Against FP64 the float centroids decide at these
distances: a centroid rounded to 6e-8 is 6e-6 of a separation of 0.01.)"""
import numpy as np
import pytest

import oracle as O
from omega3d_gb300.metrics import rel_err

pytestmark = pytest.mark.gpu


def _sphere(level, nunk):
    import omega3d_gb300 as G
    nodes, idx = G.generate_ovoid(level, 2.0, 2.0, 2.0)
    s = G.Surfaces(nodes, idx, nunk=nunk)
    rng = np.random.default_rng(level)
    ps = rng.normal(size=(3, s.npanels)).astype(np.float32)
    s.set_sheet_strengths(ps[0], ps[1], ps[2] if nunk == 3 else None)
    return s


def _shell(n, rin, rout, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(3, n))
    d /= np.linalg.norm(d, axis=0)
    return (d * rng.uniform(rin, rout, n)).astype(np.float32), rng.normal(size=(3, n)).astype(np.float32)


@pytest.mark.parametrize("level,nt,rin,rout", [(0, 1, 1.2, 1.3), (1, 33, 1.05, 1.5), (1, 200, 1.001, 1.01),
                                               (2, 65, 1.02, 3.0), (3, 31, 1.03, 1.2), (2, 1500, 1.01, 1.1)])
@pytest.mark.parametrize("maxlev", [0, 1, 3, 6])
@pytest.mark.parametrize("nunk,grads", [(2, True), (3, True), (2, False), (3, False)])
def test_panels_on_close_points(level, nt, rin, rout, maxlev, nunk, grads):
    import torch

    import omega3d_gb300 as G
    s = _sphere(level, nunk)
    x, _ = _shell(nt, rin, rout, 3)
    sss = s.ps[2] if nunk == 3 else None
    kind = "velandgrad" if grads else "velonly"
    uo, go = O.panels_affect_points(s.x, s.idx, s.area, s.ts, x, sss, grads, "rm", 1, maxlev)
    for prec in ("plain", "compensated"):
        t = G.Points(torch.from_numpy(x).cuda(), inert=True, grads=grads)
        G.panels_affect_points(s, t, G.ResultsType(kind), G.ExecEnv("rm", prec), maxlev=maxlev,
                               arrays=s.device_arrays("cuda"))
        for got, ref in ((t.u, uo),) + (((t.ug, go),) if grads else ()):
            got = got.cpu().numpy()
            assert np.isfinite(got).all()
            assert rel_err(got, ref, floor=1e-2)[0] <= 1e-5


@pytest.mark.parametrize("level,ns,rin,rout", [(0, 1, 1.2, 1.3), (1, 33, 1.05, 1.5), (1, 700, 1.001, 1.01),
                                               (2, 65, 1.02, 3.0), (3, 31, 1.03, 1.2), (2, 5000, 1.01, 1.1)])
@pytest.mark.parametrize("maxlev", [0, 1, 3, 6])
def test_close_points_on_panels(level, ns, rin, rout, maxlev):
    import torch

    import omega3d_gb300 as G
    s = _sphere(level, 2)
    x, v = _shell(ns, rin, rout, 4)
    src = G.Points(torch.from_numpy(x).cuda(), torch.from_numpy(v).cuda(), torch.full((ns,), 0.02, device="cuda"))
    po = O.points_affect_panels(x, v, s.x, s.idx, s.area, "rm", 1, maxlev)
    for prec in ("plain", "compensated"):
        pu = torch.zeros(3, s.npanels, device="cuda")
        G.points_affect_panels(src, s, G.ExecEnv("rm", prec), maxlev=maxlev, arrays=s.device_arrays("cuda"), pu=pu)
        assert rel_err(pu.cpu().numpy(), po, floor=1e-2)[0] <= 1e-5


def test_results_repeat():
    import torch

    import omega3d_gb300 as G
    s = _sphere(3, 2)
    x, v = _shell(3000, 1.01, 1.5, 9)
    arr = s.device_arrays("cuda")
    out = []
    for _ in range(3):
        t = G.Points(torch.from_numpy(x).cuda(), inert=True)
        G.panels_affect_points(s, t, G.ResultsType("velandgrad"), G.ExecEnv("rm", "compensated"), arrays=arr)
        out.append((t.u.cpu().numpy(), t.ug.cpu().numpy()))
    for u, g in out[1:]:
        assert np.array_equal(u, out[0][0]) and np.array_equal(g, out[0][1])
