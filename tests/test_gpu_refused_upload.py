"""An upload that lacks an array is refused before any host row is read: the
kernels read the rows in place, so a call that returns half-way would leave
them reading memory that the caller may release."""
import ctypes as C

import numpy as np
import pytest

import des_gb300 as D
from des_gb300 import abi, workload as W

MISSING = ["temperature", "volume_old", "stress", "shpdz", "tmp_result_sg"]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP32])
@pytest.mark.parametrize("missing", MISSING)
def test_refused_upload_changes_nothing(gpu, missing, precision):
    mesh, p, T, pls, _ = D.setup_case(W.scaled(W.CONFIGS["tiny"], 5, 4, 3))
    p.precision = precision
    dev = D.Device(mesh, p, device=0)
    dev.upload(W.new_state(mesh, T, pls), abi.F_COORD | abi.F_TEMPERATURE | abi.F_PLSTRAIN)
    dev.init_fields()
    dev.step(3)
    want = dev.download(abi.State(mesh.nnode, mesh.nelem))
    other = want.copy()
    for n in other.ARRAYS:
        getattr(other, n)[:] = 7.0
    other.time, other.dt, other.steps = 1.0, 2.0, 3
    v = other.view()
    setattr(v, missing, C.POINTER(C.c_double)())
    assert D.lib().des_gpu_upload(dev.h, C.byref(v), abi.F_ALL) == abi.DES_ERR_ARG
    got = dev.download(abi.State(mesh.nnode, mesh.nelem))
    dev.close()
    assert (got.time, got.dt, got.steps) == (want.time, want.dt, want.steps)
    for n in got.ARRAYS:
        assert np.array_equal(getattr(got, n), getattr(want, n)), n
