"""The mean density of a mix leaves absent materials out only where their term
is a zero: at an infinite temperature the reference adds inf * 0."""
import numpy as np
import pytest

from des_gb300 import abi
from helpers import Case, LOOP, phase_config


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [abi.LANES_ALONE, abi.LANES_SHARED])
@pytest.mark.parametrize("T", [np.inf, 1e306, 1e150, -1e200])
def test_hot_nodes_of_mixed_elements(gpu, T, lanes):
    c = Case(phase_config())
    em = c.mesh.elemmarkers
    em[em == 4] = 3                      # (a power of two of one material is the material's own density)
    c.oracle.set_elemmarkers(em)
    s = c.state_after(3)
    mixed = np.flatnonzero(((em > 0).sum(1) > 1) & ((em > 0).sum(1) < 3))
    assert len(mixed) > 5
    s.temperature[c.mesh.connectivity[mixed[::3], 1]] = T
    for steps in (None, 1):
        dev = c.device()
        dev.set_lanes(lanes)
        dev.upload(s)
        want = s.copy()
        if steps is None:
            for f in ("compute_mass", "update_force"):
                dev.call(f)
                c.oracle.call(f, want)
        else:
            dev.step(steps, report=False)
            c.oracle.step(want, steps)
        got = dev.download(abi.State(c.mesh.nnode, c.mesh.nelem))
        dev.close()
        assert np.isnan(want.force).any() or abs(T) < 1e300
        for f in ("mass", "tmass", "force", "vel", "temperature"):
            a, b = getattr(got, f), getattr(want, f)
            assert np.array_equal(a, b, equal_nan=True), (steps, f)
