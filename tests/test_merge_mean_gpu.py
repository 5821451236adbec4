"""GPU test of the merge's mean strength, the reference's sequential float sum, around the sizes of the
chunks it is added in (256 and 4,096 terms) and for terms whose rounding is awkward: exact ties, equal
terms, zeros first, many binades.  1,000 close pairs have strengths two float spacings apart, so
the number that merges moves when the mean is off by a few spacings; it is the oracle's."""

import numpy as np
import pytest

import omega3d_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu
PAIRS = 1000


def _terms(kind, n, rng):
    if kind == "random":
        return rng.random(n) * 1e-3
    if kind == "equal":
        return np.full(n, 0.1)
    if kind == "ties":
        return rng.integers(0, 2000, n) * 0.5
    if kind == "zeros":
        return np.where(np.arange(n) < n // 2, 0.0, rng.random(n))
    return np.exp(rng.normal(size=n) * 8.0)


@pytest.mark.parametrize("kind", ["random", "equal", "ties", "zeros", "binades"])
@pytest.mark.parametrize("n", [1, 255, 257, 4095, 4097, 50001])
def test_pairs_around_the_threshold(kind, n):
    import torch
    rng = np.random.default_rng(n)
    t = _terms(kind, n, rng).astype(np.float32)
    far = 100.0 + 10.0 * np.arange(n)
    x = np.zeros((3, n + 2 * PAIRS), np.float32)
    x[0, :n] = far
    x[1, n:] = np.repeat(10.0 * (1 + np.arange(PAIRS)), 2)
    r = np.full(n + 2 * PAIRS, 0.5, np.float32)
    x[2, n + 1::2] = 0.125                        # separation 0.125, of 1 / 3 at most
    s = np.zeros((3, n + 2 * PAIRS), np.float32)
    s[0, :n] = t
    # the pairs' strengths: around the mean of all, two spacings apart
    base = max(float(t.astype(np.float64).sum() / n), 1e-6)
    pair = (base * (1.0 + np.arange(-PAIRS // 2, PAIRS // 2) * 2.0 ** -22)).astype(np.float32)
    s[0, n:] = np.repeat(pair, 2)
    mean = np.float32(0)
    for v in s[0]:
        mean = np.float32(mean + v)
    mean = mean / np.float32(s.shape[1])
    # dist frac (strength + epsilon) < threshold mean radius / overlap, for the middle pair as an equality
    thr = float(np.float32(0.125 * 0.5 * (base + 2.0 ** -23) / (mean * np.float32(0.5) / np.float32(1.5))))
    want = O.merge_close_particles(x, s, r, 1.5, thr, False)
    d = [torch.from_numpy(a.copy()).cuda() for a in (x, s, r)]
    got = G.merge_close_particles(*d, 1.5, thr, False)
    assert got[3] == want[3]
    assert 0 < got[3] < PAIRS
