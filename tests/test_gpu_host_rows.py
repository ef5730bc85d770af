"""Uploads and downloads against host rows in place (kernels that read and write
host memory) and through the staging buffer: page-locked and ordinary arrays,
starting at every kind of place in a 128-byte line, and off a double's alignment."""
import numpy as np
import pytest

import des_gb300 as D
from des_gb300 import abi, workload as W

BOXES = [(1, 1, 1), (5, 4, 3), (13, 7, 5)]
GUARD = -7.25


def placed(mesh, offset):
    """A State whose arrays start `offset` bytes past a 128-byte line, between guards."""
    s, whole = abi.State(mesh.nnode, mesh.nelem), {}
    for n in s.ARRAYS:
        a = getattr(s, n)
        raw = np.zeros(a.nbytes + 512, np.uint8)
        at = -raw.ctypes.data % 128 + 128 + offset
        view = raw[at - 16:at + a.nbytes + 16].view(np.float64)
        view[:] = GUARD
        whole[n] = view
        setattr(s, n, view[2:-2].reshape(a.shape))
    return s, whole


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP32])
@pytest.mark.parametrize("box", BOXES)
def test_rows_at_any_place(gpu, box, precision):
    cfg = W.scaled(W.CONFIGS["tiny"], *box)
    mesh, p, T, pls, _ = D.setup_case(cfg)
    p.precision = precision
    dev = D.Device(mesh, p, device=0)
    dev.upload(W.new_state(mesh, T, pls), abi.F_COORD | abi.F_TEMPERATURE | abi.F_PLSTRAIN)
    dev.init_fields()
    dev.step(3)
    want = dev.download(abi.State(mesh.nnode, mesh.nelem))
    for offset in (0, 8, 16, 120, 4):              # 4: the staging buffer
        for locked in (False, True):
            s, whole = placed(mesh, offset)
            if locked:
                D.pin(s)
            dev.download(s)
            for n in s.ARRAYS:
                assert np.array_equal(getattr(s, n), getattr(want, n)), (n, offset, locked)
                assert (whole[n][:2] == GUARD).all() and (whole[n][-2:] == GUARD).all(), (n, offset, locked)
            other = D.Device(mesh, p, device=0)
            other.upload(s)
            back = other.download(abi.State(mesh.nnode, mesh.nelem))
            other.close()
            if locked:
                D.unpin(s)
            for n in s.ARRAYS:
                # (the FP32 form's stress is split anew on upload)
                if n == "stress" and precision == abi.PREC_FP32:
                    assert np.allclose(back.stress, want.stress, rtol=2.0 ** -23, atol=2.0 ** -23 * np.abs(want.stress).max())
                else:
                    assert np.array_equal(getattr(back, n), getattr(want, n)), (n, offset, locked)
    dev.close()
