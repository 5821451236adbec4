"""CPU emulation of the panel kernels' node queue (take_nodes in o3g_panel.cu): 32 nodes are taken
from its end, those that split push their children behind what is left, child by child.  Its length must stay
within queue_cap(tpt, maxlev) = 31 + 64 tpt + 96 (maxlev - 1) + 128 whatever splits: everything, nothing,
at random, and what was taken from the shallow end of a mixed batch only."""
import numpy as np
import pytest


def queue_cap(tpt, maxlev):
    return 31 + 64 * tpt + 96 * max(maxlev - 1, 0) + 128


def _longest(tpt, maxlev, decide, rng, steps=40):
    q, longest = [], 0
    for step in range(steps):
        q += [0] * int(rng.integers(0, 64 * tpt + 1) if step else 64 * tpt)   # a sweep step's near pairs
        longest = max(longest, len(q))
        while len(q) >= 32:
            batch, q = q[-32:], q[:-32]
            split = [lev for lev, s in zip(batch, decide(batch)) if s and lev < maxlev]
            q += [lev + 1 for _ in range(4) for lev in split]
            longest = max(longest, len(q))
    return longest


@pytest.mark.parametrize("tpt", [1, 2])
@pytest.mark.parametrize("maxlev", range(7))
def test_queue_stays_within_its_capacity(tpt, maxlev):
    rng = np.random.default_rng(10 * maxlev + tpt)
    rules = [lambda b: [True] * len(b), lambda b: [False] * len(b)]
    for p in (0.1, 0.3, 0.6, 0.9, 0.97):
        rules.append(lambda b, p=p: rng.random(len(b)) < p)
    rules.append(lambda b: [lev == min(b) for lev in b])
    rules.append(lambda b: [lev == max(b) for lev in b])
    for r in rules:
        steps = 4 if maxlev > 3 else 20
        assert _longest(tpt, maxlev, r, rng, steps) <= queue_cap(tpt, maxlev)
