"""Both forms of the step's kernels (one thread per node and element, which
real meshes run, and shared lanes, which every box of these sizes would run
by its size) on the same meshes: the same bits from both, over the option
variants and the yielding, layered and visco-plastic boxes, in both
precisions; and against the oracle where an operand leaves the integer pipes'
range or a node's support list is longer than a chunk."""
import numpy as np
import pytest

import des_gb300 as D
from des_gb300 import abi, workload as W
from helpers import (Case, COMPARED, OPTION_TRANSCENDENTAL, OPTION_VARIANTS, evp_config, layered_config, phase_config,
                     plastic_config, rel_l2)
from oracle.oracle import PortOracle

pytestmark = pytest.mark.gpu
BOTH = (abi.LANES_ALONE, abi.LANES_SHARED)
CONFIGS = dict(OPTION_VARIANTS, plastic=plastic_config(), evp=evp_config(), layered=layered_config(), phase=phase_config(),
               yielding=W.scaled(W.CONFIGS["yield"], 9, 7, 5),
               evp_yielding=W.scaled(W.CONFIGS["yield"], 7, 5, 4))
CONFIGS["evp_yielding"].rheology = "evp"
_cases = {}


def case(name):
    if name not in _cases:
        _cases[name] = Case(CONFIGS[name])
    return _cases[name]


def run(mesh, params, start, nsteps, lanes, mask=abi.F_ALL, init=False, host=False):
    dev = D.Device(mesh, params, device=0)
    dev.set_lanes(lanes)
    s = start.copy()
    dev.upload(s, mask)
    if init:
        dev.init_fields()
    rep = None
    for n in nsteps:
        rep = dev.step_host(s, n) if host else dev.step(n)
    kernels = dev.kernels_per_step
    got = dev.download(abi.State(mesh.nnode, mesh.nelem))
    dev.close()
    return got, rep, kernels


def same(a, b, fields=None):
    for f in fields or COMPARED + ["coord0"]:
        assert np.array_equal(getattr(a, f), getattr(b, f), equal_nan=True), f
    assert (a.time, a.dt, a.steps) == (b.time, b.dt, b.steps)


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP32])
@pytest.mark.parametrize("name", sorted(CONFIGS))
def test_same_bits_from_both_forms(name, precision):
    c = case(name)
    p = abi.Params.from_buffer_copy(c.params)
    p.precision = precision
    s = W.new_state(c.mesh, c.T, c.pls)
    mask = abi.F_COORD | abi.F_TEMPERATURE | abi.F_PLSTRAIN
    (a, ra, ka), (b, rb, kb) = (run(c.mesh, p, s, (3, 47, 40), lanes, mask, init=True) for lanes in BOTH)
    same(a, b)
    assert ra.status == rb.status and ra.eigen_solves == rb.eigen_solves and ra.exact_returns == rb.exact_returns
    # the forms did differ: E-A's three kernels, and the FP32 list of exact returns
    plastic = p.rheol_type in (abi.RH_EP, abi.RH_EVP)
    assert ka - kb == ((2 if p.has_thermal_diffusion else 1) if precision == abi.PREC_FP64 else int(plastic))
    if name in ("plastic", "yielding", "evp_yielding"):
        assert ra.eigen_solves > 0 and (precision == abi.PREC_FP64 or ra.exact_returns > 0)


@pytest.mark.parametrize("lanes", BOTH)
@pytest.mark.parametrize("name", sorted(set(CONFIGS) - OPTION_TRANSCENDENTAL - {"plastic", "yielding", "evp", "evp_yielding", "layered"}))
def test_both_forms_equal_the_oracle(name, lanes):
    """(variants without CUDA's own transcendentals: every bit)"""
    c = case(name)
    s = c.initial_state()
    got, rep, _ = run(c.mesh, c.params, s, (30,), lanes)
    want = s.copy()
    c.oracle.step(want, 30)
    same(got, want, COMPARED)


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP32])
@pytest.mark.parametrize("name", ["free_x0", "phase", "yielding"])
def test_host_steps_in_both_forms(name, precision):
    c = case(name)
    p = abi.Params.from_buffer_copy(c.params)
    p.precision = precision
    s = c.state_after(11)
    (a, _, _), (b, _, _) = (run(c.mesh, p, s, (1, 1, 3), lanes, host=True) for lanes in BOTH)
    same(a, b)


def out_of_range(s, mesh, what):
    if what == "stress":                 # 1e-300 Pa, subnormal strain, slow nodes
        s.stress[::7, 3:] = 1e-300
        s.strain[::5, 3:] = 5e-324
        s.vel[::3, 1] = 1e-290
    elif what == "forces":               # the force sums cancel to 0 or are below 2^-900
        s.stress[:] = 0
        s.stress[::3, 0] = 1e-295
        s.stress[1::9, 3] = -1e-280
        s.vel[:] = 0
    elif what == "coordinates":          # edge components of 1e-200 and 5e-324 m
        x0 = np.flatnonzero(s.coord[:, 0] == s.coord[:, 0].min())
        s.coord[x0, 0] = 0
        s.coord[x0[1::3], 0] = 1e-200
        s.coord[x0[2::3], 0] = 5e-324
    elif what == "volumes":              # slivers: volumes far below their neighbours'
        for e in range(0, mesh.nelem, 37):
            n = mesh.connectivity[e]
            centre = s.coord[n[1:]].mean(0)
            if s.mass[n[0]] > 0:
                s.coord[n[0]] = centre + (s.coord[n[0]] - centre) * 2.0 ** -14
                s.mass[mesh.connectivity[(mesh.connectivity == n[0]).any(1)].ravel()] = -1   # one move a neighbourhood


@pytest.mark.parametrize("lanes", BOTH)
@pytest.mark.parametrize("what", ["stress", "forces", "coordinates", "volumes"])
def test_operands_out_of_range(what, lanes):
    c = case("no_gravity" if what == "forces" else "elastic_fnd" if what == "coordinates" else "phase")
    s = c.state_after(3)
    out_of_range(s, c.mesh, what)
    if what in ("coordinates", "volumes"):
        s.volume_old[:] = s.volume
        for f in ("compute_volume", "compute_mass", "compute_shape_fn"):
            c.oracle.call(f, s)
        # (the moved nodes turn some elements inside out; the loop does not mind)
        s.dt *= 1e-3
    got, _, _ = run(c.mesh, c.params, s, (2,), lanes)
    want = s.copy()
    c.oracle.step(want, 2)
    for f in COMPARED:
        assert np.array_equal(getattr(got, f), getattr(want, f), equal_nan=True), f


@pytest.mark.parametrize("what", ["stress", "forces", "coordinates", "volumes"])
def test_operands_out_of_range_fp32(what):
    c = case("elastic_fnd" if what == "coordinates" else "phase")
    s = c.state_after(3)
    out_of_range(s, c.mesh, what)
    if what in ("coordinates", "volumes"):
        for f in ("compute_volume", "compute_mass", "compute_shape_fn"):
            c.oracle.call(f, s)
        s.dt *= 1e-3
    p = abi.Params.from_buffer_copy(c.params)
    p.precision = abi.PREC_FP32
    (a, _, _), (b, _, _) = (run(c.mesh, p, s, (2,), lanes) for lanes in BOTH)
    same(a, b)


class Ball:
    """A box's surface grid joined to one node inside: 12 m m tets share it.  Fields as workload.Mesh."""

    def __init__(self, m, lx=40e3, ly=30e3, lz=20e3):
        rng = np.random.default_rng(m)
        node, tri = {}, []
        side = lambda k, i, j, hi: {0: (hi * m, i, j), 1: (i, hi * m, j), 2: (i, j, hi * m)}[k]  # noqa: E731
        for k in range(3):
            for hi in range(2):
                for i in range(m):
                    for j in range(m):
                        q = [side(k, i + a, j + b, hi) for a, b in ((0, 0), (1, 0), (1, 1), (0, 1))]
                        for t in ((0, 1, 2), (0, 2, 3)):
                            tri.append(([q[v] for v in t], 1 << (2 * k + hi)))
        for t, _ in tri:
            for v in t:
                node.setdefault(v, len(node))
        self.nnode, self.nelem, self.nseg, self.nmat = len(node) + 1, len(tri), len(tri), 1
        self.coord = np.zeros((self.nnode, 3))
        for v, k in node.items():
            self.coord[k] = np.array(v) / m * (lx, ly, lz) - (0, 0, lz)
        self.coord[-1] = (0.47 * lx, 0.52 * ly, -0.55 * lz)
        self.connectivity = np.zeros((self.nelem, 4), np.int32)
        self.segment = np.zeros((self.nseg, 3), np.int32)
        self.segflag = np.array([f for _, f in tri], np.int32)
        for e, (t, _) in enumerate(tri):
            n = [node[v] for v in t]
            a, b, c = self.coord[n]
            if np.dot(np.cross(b - a, c - a), self.coord[-1] - a) < 0:
                n[1], n[2] = n[2], n[1]
            # a positive volume in the order of the library's own boxes: node 3 to the left of 0 1 2
            self.connectivity[e] = (n[0], n[1], n[2], self.nnode - 1)
            self.segment[e] = n
        order = rng.permutation(self.nelem)
        self.connectivity = np.ascontiguousarray(self.connectivity[order])
        self.elemmarkers = np.full((self.nelem, 1), 4, np.int32)

    view = W.Mesh.view


# 12 m m tets around the middle node: 48 (one chunk of 32 and a half), 108 (three
# chunks and 12), 300; the surface's nodes have 4 to 8
@pytest.mark.parametrize("m", [2, 3, 5])
def test_support_lists_longer_than_a_chunk(m):
    mesh = Ball(m)
    cfg = W.scaled(W.CONFIGS["1"], m, m, m)
    _, p, _, _, _ = D.setup_case(cfg)
    p.zlength = 20e3
    p.compensation_pressure = p.rho0.v[0] * p.gravity * p.zlength
    T = 273.0 + 1300.0 * -mesh.coord[:, 2] / 20e3 + np.random.default_rng(m).normal(0, 5, mesh.nnode)
    ref = W.new_state(mesh, T, np.zeros(mesh.nelem))
    o = PortOracle(mesh, p)
    o.init_fields(ref)
    assert (ref.volume > 0).all() and np.bincount(mesh.connectivity.ravel()).max() == 12 * m * m
    start = ref.copy()
    o.step(ref, 23)
    for lanes in BOTH:
        got, _, _ = run(mesh, p, start, (3, 20), lanes)
        same(got, ref, COMPARED)
    p.precision = abi.PREC_FP32
    (a, _, _), (b, _, _) = (run(mesh, p, start, (3, 20), lanes) for lanes in BOTH)
    same(a, b)
    one = start.copy()
    o.step(one, 1)
    got, _, _ = run(mesh, p, start, (1,), abi.LANES_SHARED)
    for f in ("force", "stress", "strain", "mass", "tmass", "volume_n"):
        assert rel_l2(getattr(got, f), getattr(one, f)) <= 1e-6, f
