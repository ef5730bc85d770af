"""The FP32 estimate that decides whether a power-law viscosity is clipped:
elements within a few per cent of a clip take the FP64 value, and an absent material
whose law does not give a positive number (the reference divides its count of 0
by a viscosity of 0) is not left out of a mix."""
import numpy as np
import pytest

from des_gb300 import workload as W
from helpers import Case, layered_config, rel_l2

pytestmark = pytest.mark.gpu
FIELDS = ["stress", "strain", "strain_rate", "plstrain", "dpressure"]


def with_params(cfg, mats=None, **params):
    d = dict(cfg.__dict__)
    d["extra"] = dict(cfg.extra, params=dict(cfg.extra.get("params", {}), **params), mats=dict(cfg.extra.get("mats", {}), **(mats or {})))
    return W.Config(**d)


def update_stress(c, steps=7):
    s = c.state_before("update_stress", steps)
    want = s.copy()
    c.oracle.call("update_stress", want)
    dev = c.device()
    dev.upload(s)
    dev.call("update_stress")
    got = dev.download(s.copy())
    dev.close()
    return got, want


def viscosity(c, s):
    """matprops.cxx:607-643 before the clip, one material, from the corrected strain rate."""
    P, e = c.params, s.strain_rate
    T = s.temperature[c.mesh.connectivity].mean(1)
    a = e[:, :3].mean(1)
    e2 = np.maximum(np.sqrt(0.5 * ((e[:, :3] - a[:, None]) ** 2).sum(1) + (e[:, 3:] ** 2).sum(1)), 1e-30)
    n = P.visc_exponent.v[0]
    return (0.25 * e2 ** (1 / n - 1) * (0.75 * P.visc_coefficient.v[0]) ** (-1 / n) *
            np.exp(P.visc_activation_energy.v[0] / (n * 8.3144 * T)) * 1e6)


@pytest.mark.parametrize("end", ["visc_min", "visc_max"])
def test_elements_at_the_clip(gpu, end):
    base = W.scaled(W.CONFIGS["3"], 20, 20, 8)
    maxwell = dict(rheol_type=3, visc_min=1e16, visc_max=1e30)
    c = Case(with_params(base, **maxwell))
    _, want = update_stress(c)
    near = float(np.median(viscosity(c, want)))
    # the time step follows visc_min, so the state is the run's with the new clip
    c = Case(with_params(base, **dict(maxwell, **{end: near})))
    got, want = update_stress(c)
    r = viscosity(c, want) / near
    assert ((r > 0.93) & (r < 1.07)).sum() > 10
    assert (r < 1).any() and (r > 1).any()
    for f in FIELDS:
        assert rel_l2(getattr(got, f), getattr(want, f)) <= 1e-12, f
    # element by element: a wrong clip moves one stress by per cents
    err = np.abs(got.stress - want.stress).max(1) / np.abs(want.stress).max(1)
    assert err.max() <= 1e-11


def test_a_law_without_a_viscosity(gpu):
    """Material 2's coefficient to the power -2 underflows to 0: where it is
    absent from a mix of materials 0 and 1, its term is 0 / 0 in the reference
    and the Maxwell stress is never taken."""
    c = Case(with_params(layered_config(12, 10, 10), mats=dict(visc_exponent=[3.5, 3.5, 0.5], visc_coefficient=[7e4, 7e4, 1e300]),
                         visc_max=1e20))
    em = c.mesh.elemmarkers
    mixed = (em[:, 0] > 0) & (em[:, 1] > 0) & (em[:, 2] == 0)
    assert mixed.sum() > 20
    got, want = update_stress(c)
    err = np.abs(got.stress - want.stress).max(1) / np.abs(want.stress).max(1)
    assert err[mixed].max() <= 1e-11
