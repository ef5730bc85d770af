"""Forward passes whose output rows lie over their input rows (a caller's own
workspace): the same values as with rows of their own, whatever the distance
between the two."""
import ctypes as C

import numpy as np
import pytest

import des_gb300 as D
from des_gb300 import abi, closure

FP = C.POINTER(C.c_float)


# 40,000 samples: more tiles than the GPU has multiprocessors, so that a tile's
# outputs fall on the inputs of tiles that start later.  Offsets in floats: y at
# x, inside it, half before it, over its last rows (8: not one row of x, 3: off
# the 16-byte alignment).
@pytest.mark.gpu
@pytest.mark.parametrize("n,at", [(1, 0), (300, 0), (40000, 0), (40000, 8), (40000, 3), (40000, -160000), (40000, 639992)])
def test_outputs_over_inputs(gpu, n, at):
    rng = np.random.default_rng(n)
    x = np.zeros((n, 16), np.float32)
    x[:, :14] = rng.normal(0, 1, (n, 14))
    net = closure.new_net(3)
    want = closure.forward(net, x)
    work = np.zeros(64 + max(-at, 0) + 16 * n + 8 * n, np.float32)
    base = (-work.ctypes.data // 4) % 4 + max(-at, 0)
    xs, ys = work[base:base + 16 * n], work[base + at:base + at + 8 * n]
    xs[:] = x.ravel()
    rc = D.lib().des_mlp_forward(C.byref(net), xs.ctypes.data_as(FP), n, ys.ctypes.data_as(FP))
    assert rc == abi.DES_OK
    assert np.array_equal(ys.reshape(n, 8), want)
