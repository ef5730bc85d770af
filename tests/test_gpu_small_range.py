"""Rates below the normal range in the four-lane E-A: with velocities so small
that the products leave the integer pipes' range, half the sum of the spin's
and strain rate's brackets is not the sum of their halves, and the element is
formed as the reference forms it."""
import numpy as np
import pytest

from des_gb300 import abi
from helpers import Case, COMPARED, OPTION_VARIANTS


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-304, 1e-308])
def test_subnormal_rates(gpu, scale):
    c = Case(OPTION_VARIANTS["no_gravity"])
    s = c.state_after(3)
    rng = np.random.default_rng(5)
    s.stress[:] = 0
    s.vel[:] = scale * rng.normal(0, 1, s.vel.shape)
    want = s.copy()
    c.oracle.step(want, 2)
    # (the first step's velocities give the second's rates; the moved sides' are ordinary)
    assert (np.abs(want.strain_rate[want.strain_rate != 0]).min()) < 2.3e-308
    dev = c.device()
    dev.upload(s)
    dev.step(2)
    got = dev.download(abi.State(c.mesh.nnode, c.mesh.nelem))
    dev.close()
    for f in COMPARED:
        assert np.array_equal(getattr(got, f), getattr(want, f)), f
