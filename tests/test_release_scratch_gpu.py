"""The scratch that a particle split keeps for the next one goes back to the device on
o3g_release_scratch, and the next split gives the same bits."""
import numpy as np
import pytest

import omega3d_gb300 as G
from omega3d_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_released_after_a_split(cuda):
    import torch
    x, s, r, e = (torch.from_numpy(a).cuda() for a in W.lattice_particles(k=64, seed=3))

    def free():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    def run():
        out = G.split_elongated(x, s, r, e)
        return [t.cpu().numpy().view(np.uint32) for t in out[:4]]

    run()                                  # (kernels and their local memory are loaded for good)
    G.release_scratch()
    before = free()
    a = run()
    assert before - free() > 64 << 20      # 262,144 particles: some 200 MB are kept
    G.release_scratch()
    assert before - free() < 32 << 20      # (allocation granularity)
    b = run()
    assert all(np.array_equal(p, q) for p, q in zip(a, b))
    G.release_scratch()
    G.release_scratch()
    assert before - free() < 32 << 20
