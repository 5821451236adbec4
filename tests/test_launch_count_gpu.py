"""o3g_launch_count over a factorisation: the kernels launched, counted by hand for small systems.
n <= 64: one panel and the diagonal inverses.  n <= 128: two panels of 64 columns, the update between them,
two row interchanges, the inverses.  n = 200: four panels, two updates between, four interchanges, the
block solve, the tensor-core update (two kernels), the inverses and one merge of them."""
import ctypes

import numpy as np
import pytest

import omega3d_gb300 as G
from omega3d_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,launches", [(20, 2), (64, 2), (100, 6), (128, 6), (200, 15)])
def test_factorisation(n, launches, cuda):
    bem = G.BEM(n)
    bem.set_block(0, 0, np.eye(n, dtype=np.float32))
    c = [ctypes.c_uint64(), ctypes.c_uint64()]
    L.check(L.lib().o3g_launch_count(ctypes.byref(c[0])), "count")
    bem.factor()
    L.check(L.lib().o3g_launch_count(ctypes.byref(c[1])), "count")
    assert c[1].value - c[0].value == launches
