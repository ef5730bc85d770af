"""The kernels that share a node between eight lanes and an element between
four (csrc/des_small.cuh) against the oracle on the smallest meshes and at the
remainders of their tiles, and against the one-thread kernels' route on a mesh
above every crossing point (one box, both sides of it, in test_gpu_step.py and
test_gpu_fullsize.py)."""
import numpy as np
import pytest

import des_gb300 as D
from des_gb300 import abi, workload as W
from helpers import rel_l2
from oracle.oracle import PortOracle

FIELDS = ["coord", "vel", "force", "temperature", "mass", "tmass", "volume_n", "ntmp", "volume", "volume_old",
          "edvoldt", "plstrain", "dpressure", "stress", "strain", "strain_rate", "shpdx", "shpdy", "shpdz"]

# 6 elements (less than a block of quads), 8 nodes (less than a block of
# octets), one element over and under a block, a support list of 24 and more
# than one chunk's rest, a dt step within the run, a zero velocity component
BOXES = [(1, 1, 1), (2, 1, 1), (1, 1, 11), (3, 3, 3), (7, 5, 3), (11, 9, 5)]


@pytest.mark.gpu
@pytest.mark.parametrize("box", BOXES)
def test_small_meshes_bit_identical(gpu, box):
    cfg = W.scaled(W.CONFIGS["tiny"], *box)
    mesh, p, T, pls, _ = D.setup_case(cfg)
    ref, s = W.new_state(mesh, T, pls), W.new_state(mesh, T, pls)
    o = PortOracle(mesh, p)
    o.init_fields(ref)
    dev = D.Device(mesh, p, device=0)
    dev.upload(s, abi.F_COORD | abi.F_TEMPERATURE | abi.F_PLSTRAIN)
    dev.init_fields()
    for n in (1, 2, 20, 47):               # single-step graphs, then ten steps to a graph
        o.step(ref, n)
        dev.step(n)
        got = dev.download(abi.State(mesh.nnode, mesh.nelem), abi.F_STEP_STATE)
        for f in FIELDS:
            assert np.array_equal(getattr(got, f), getattr(ref, f)), (n, f)
        assert got.dt == ref.dt and got.time == ref.time and got.steps == ref.steps
    dev.close()


@pytest.mark.gpu
@pytest.mark.parametrize("box", [(5, 4, 3), (24, 24, 14)])     # lanes shared; one thread each
def test_operands_out_of_range_take_the_exact_path(gpu, box):
    """Stress of 1e-300 Pa and velocities of 1e-290 m/s in a few elements: their
    products leave the integer pipes' range, the result must not change."""
    cfg = W.scaled(W.CONFIGS["tiny"], *box)
    mesh, p, T, pls, _ = D.setup_case(cfg)
    ref = W.new_state(mesh, T, pls)
    o = PortOracle(mesh, p)
    o.init_fields(ref)
    o.step(ref, 3)
    ref.stress[::7, 3:] = 1e-300
    ref.strain[::5, 3:] = 5e-324
    ref.vel[::3, 1] = 1e-290
    dev = D.Device(mesh, p, device=0)
    dev.upload(ref, abi.F_ALL)
    o.step(ref, 2)
    dev.step(2)
    got = dev.download(abi.State(mesh.nnode, mesh.nelem), abi.F_STEP_STATE)
    for f in FIELDS:
        assert np.array_equal(getattr(got, f), getattr(ref, f)), f
    dev.close()


@pytest.mark.gpu
@pytest.mark.parametrize("box", BOXES)
def test_small_meshes_fp32(gpu, box):
    """The FP32 form's shared-lane kernels: one step from the oracle's state to
    the one-step bars of test_gpu_fp32.py, and the temperature (1e-12 there)
    after a second step, which is the first to read the pass's conduction."""
    cfg = W.scaled(W.CONFIGS["tiny"], *box)
    mesh, p, T, pls, _ = D.setup_case(cfg)
    ref = W.new_state(mesh, T, pls)
    o = PortOracle(mesh, p)
    o.init_fields(ref)
    o.step(ref, 9)                         # the step after it forms dt
    p32 = abi.Params.from_buffer_copy(p)
    p32.precision = abi.PREC_FP32
    dev = D.Device(mesh, p32, device=0)
    dev.upload(ref, abi.F_ALL)
    o.step(ref, 1)
    dev.step(1)
    got = dev.download(abi.State(mesh.nnode, mesh.nelem), abi.F_STEP_STATE)
    for f in ["vel", "force", "stress", "strain", "mass", "tmass", "volume_n", "volume", "shpdx", "shpdy", "shpdz"]:
        assert rel_l2(getattr(got, f), getattr(ref, f)) <= 1e-6, f
    assert got.dt == pytest.approx(ref.dt, rel=1e-6) and got.steps == ref.steps
    o.step(ref, 1)
    dev.step(1)
    dev.download(got, abi.F_STEP_STATE)
    assert rel_l2(got.temperature, ref.temperature) <= 1e-12
    dev.close()
