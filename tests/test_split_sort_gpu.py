"""The particle split where its neighbour sort changes form: clusters of up to 32, 128, 256 and more
particles, all of them elongated and within each other's search radius, so that every particle's
list has the cluster's size.  Bit for bit the oracle's."""

import numpy as np
import pytest

import omega3d_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 2, 31, 32, 33), (63, 64, 65, 127, 128), (129, 255, 256, 257), (300, 513)])
def test_cluster_sizes(sizes):
    import torch
    rng = np.random.default_rng(sum(sizes))
    n = sum(sizes)
    at = np.repeat(10.0 * np.arange(len(sizes)), sizes)
    x = rng.uniform(-0.2, 0.2, (3, n))
    x[0] += at
    order = rng.permutation(n)          # the clusters' indices interleave
    x = x[:, order].astype(np.float32)
    s = (rng.normal(size=(3, n)) * 1e-2 + 0.02).astype(np.float32)
    r = rng.uniform(0.4, 0.5, n).astype(np.float32)      # search radius 3 r / 1.5, cluster diameter 0.7
    e = np.full(n, 1.5, np.float32)
    want = O.split_elongated(x, s, r, e, 0, 1.5, 1.2)
    got = G.split_elongated(*(torch.from_numpy(a.copy()).cuda() for a in (x, s, r, e)), "gaussian", 1.5, 1.2)
    assert got[4] == want[4] == n
    for a, b in zip(got[:4], want[:4]):
        assert np.array_equal(a.cpu().numpy().view(np.uint32), np.ascontiguousarray(b, np.float32).view(np.uint32))
