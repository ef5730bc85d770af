"""Downloads into, and uploads and forward passes from and into, ordinary arrays
whose pages nobody has touched yet, wholly or in part: the same values as in
arrays that were written before."""
import mmap

import numpy as np
import pytest

import des_gb300 as D
from des_gb300 import abi, closure, workload as W

pytestmark = pytest.mark.gpu


def untouched(shape, dtype, first=0):
    """A zero array in its own fresh mapping, with its first entries written."""
    n = int(np.prod(shape))
    a = np.frombuffer(mmap.mmap(-1, n * np.dtype(dtype).itemsize), dtype)
    a[:first] = 0
    return a.reshape(shape)


def state(mesh, part):
    s = abi.State(mesh.nnode, mesh.nelem)
    for n in s.ARRAYS:
        a = getattr(s, n)
        setattr(s, n, untouched(a.shape, np.float64, int(part * a.size)))
    return s


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP32])
def test_transfers(gpu, precision):
    mesh, p, T, pls, _ = D.setup_case(W.scaled(W.CONFIGS["tiny"], 40, 40, 20))     # stress: 9.2 MB
    p.precision = precision
    dev = D.Device(mesh, p, device=0)
    dev.upload(W.new_state(mesh, T, pls), abi.F_COORD | abi.F_TEMPERATURE | abi.F_PLSTRAIN)
    dev.init_fields()
    dev.step(3)
    want = abi.State(mesh.nnode, mesh.nelem)
    for n in want.ARRAYS:
        getattr(want, n)[:] = 1.0
    dev.download(want)
    for part in (0.0, 0.5):
        got = dev.download(state(mesh, part))
        for n in got.ARRAYS:
            assert np.array_equal(getattr(got, n), getattr(want, n)), (n, part)
        other = D.Device(mesh, p, device=0)
        other.upload(want)
        other.upload(state(mesh, part))           # zeros over everything
        back = other.download(abi.State(mesh.nnode, mesh.nelem))
        other.close()
        for n in back.ARRAYS:
            assert not getattr(back, n).any(), (n, part)
    dev.close()


@pytest.mark.parametrize("n", [40000, 250007])
def test_closure_outputs(gpu, n):
    rng = np.random.default_rng(n)
    x = rng.normal(0, 1, (n, 16)).astype(np.float32)
    x[:, 14:] = 0
    net = closure.new_net(1)
    want = np.ones((n, 8), np.float32)
    fp = closure._fptr
    for y in (want, untouched((n, 8), np.float32), untouched((n, 8), np.float32, 4 * n)):
        assert D.lib().des_mlp_forward(net, fp(x), n, fp(y)) == abi.DES_OK
        assert np.array_equal(y, want)
    zeros = closure.forward(net, np.zeros((n, 16), np.float32) + 0.0)
    assert np.array_equal(closure.forward(net, untouched((n, 16), np.float32)), zeros)
