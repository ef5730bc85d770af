"""The closure's rows in host memory: read and written in place where they are
16-byte aligned, through a device copy where they are not; the same results
either way, over tile remainders and from several threads."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from des_gb300 import abi, closure

pytestmark = pytest.mark.gpu
WEIGHTS = ("w1", "b1", "w2", "b2", "w3", "b3")


def _shifted(a, k):
    """A copy of a that starts 4 k bytes past a 16-byte boundary."""
    flat = np.zeros(a.size + 8, np.float32)
    off = (-flat.ctypes.data // 4) % 4 + k
    v = flat[off:off + a.size].reshape(a.shape)
    v[:] = a
    assert v.ctypes.data % 16 == 4 * k
    return v


def _case(n):
    rng = np.random.default_rng(n)
    x, t = rng.normal(0, 1, (n, 16)).astype(np.float32), rng.normal(0, 1, (n, 8)).astype(np.float32)
    x[:, 14:] = 0
    t[:, 7:] = 0
    return closure.new_net(n), x, t


@pytest.mark.parametrize("n", [1, 127, 129, 19457, 40000])
def test_rows_in_place_and_copied_agree(gpu, n):
    net, x, t = _case(n)
    y = closure.forward(net, _shifted(x, 0))
    loss, g = closure.loss_grad(net, _shifted(x, 0), _shifted(t, 0))
    for k in (1, 2):
        assert np.array_equal(closure.forward(net, _shifted(x, k)), y)
        l2, g2 = closure.loss_grad(net, _shifted(x, k), _shifted(t, k))
        # FP32 sums of 128-sample tiles added by atomics in any order: the
        # largest term times a few roundings
        assert abs(l2 - loss) <= 1e-6 * loss
        for w in WEIGHTS:
            a, b = g.arr(w), g2.arr(w)
            assert np.abs(a - b).max() <= 1e-5 * np.abs(a).max()


def test_calls_from_several_threads(gpu):
    cases = [_case(n) for n in (300, 5000, 129, 2000)]
    want = [closure.forward(net, x) for net, x, _ in cases]
    with ThreadPoolExecutor(4) as ex:
        for _ in range(3):
            got = list(ex.map(lambda c: closure.forward(c[0], c[1]), cases))
            assert all(np.array_equal(a, b) for a, b in zip(got, want))
