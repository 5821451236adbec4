"""clear_inner_layer where its kernel skips panels: bit for bit the oracle's, for points near, around and
very far from the body (beyond the reference's cap of 9.9e9 on a squared distance all panels tie),
numbers of points and panels around a warp, a block and a tile, and normals that are not unit or not
perpendicular, whose panels may never be skipped."""

import numpy as np
import pytest

import omega3d_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu


def _points(n, rng):
    d = rng.normal(size=(3, n))
    d /= np.linalg.norm(d, axis=0)
    r = np.concatenate([rng.uniform(0.9, 1.1, n), rng.uniform(0.0, 3.0, n), 10.0 ** rng.uniform(0.0, 7.0, n)])
    return (d * rng.permutation(r)[:n]).astype(np.float32)


@pytest.mark.parametrize("normals", ["true", "long", "tilted", "mixed"])
@pytest.mark.parametrize("n,level,keep", [(1, 1, 80), (33, 1, 3), (129, 2, 320), (3000, 3, 1277)])
def test_bit_exact(n, level, keep, normals):
    import torch
    rng = np.random.default_rng(n)
    nodes, idx = G.generate_ovoid(level, 2.0, 2.0, 2.0)
    idx = np.asarray(idx, np.uint32).reshape(-1, 3)[:keep].ravel().copy()
    s = G.Surfaces(np.asarray(nodes, np.float32), idx, nunk=2)
    norm = np.asarray(s.norm).copy()
    if normals == "long":
        norm *= np.float32(1.5)
    if normals in ("tilted", "mixed"):
        t = (norm + rng.normal(size=norm.shape) * 0.3).astype(np.float32)
        pick = rng.random(norm.shape[1]) < (1.0 if normals == "tilted" else 0.1)
        norm[:, pick] = t[:, pick]
    s.norm[...] = norm
    x = _points(n, rng)
    for ips in (0.02, 0.5):
        want = x.copy()
        no = O.clear_inner_layer(want, s.x, s.idx, s.norm, ips=ips)
        X = torch.from_numpy(x.copy()).cuda()
        ng = G.clear_inner_layer(s, G.Points(X, None, None, inert=True), ips=ips)
        assert ng == no
        assert np.array_equal(X.cpu().numpy().view(np.uint32), want.view(np.uint32))
