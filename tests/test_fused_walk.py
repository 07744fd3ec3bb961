"""The fused step over walks of any length.

A block of the fused pass walks its tile plane by plane; the plan picks the length from the grids'
sizes, which gives small meshes one plane a walk.  LBFS_GRID_WALK sets it, so that what a walk carries
between planes (the ring of staged planes and viscosity factors, staged ghost records, the states two
planes down, the open sums) is reached at sizes with partial tiles and on every kind of end.  Results
do not depend on the walk, bit for bit, and agree with the separate kernels to the parity bound.
"""
import numpy as np
import pytest

from helpers import FP64_RTOL, rel_err
from lbfs_b200 import GpuSolver, StepParams, _abi, build_uniform_mesh, cases
from lbfs_b200.ensemble import concatenate

pytestmark = pytest.mark.gpu

WALL, OPEN, PERIODIC = (2, 1, 1.0, 0.0, 0.0, 0.0), (2, 2, 1.0, 0.0, 0.0, 0.0), (3, 3, 1.0, 0.0, 0.0, 0.0)
MOVING, PRESSURE = (2, 1, 1.0, 0.004, 0.001, -0.002), (1, 2, 1.001, 0.0, 0.0, 0.0)
INLET, SHEAR = (2, 9, 1.0, 1e-5, 0.0, 0.0), (2, 10, 1.0, 1e-4, 0.0, 0.0)
SIDES = ("left", "right", "bottom", "top", "back", "front")
ENDS = {  # -x, +x, -y, +y, -z, +z
    "open_z": (WALL, MOVING, WALL, MOVING, OPEN, OPEN),
    "walls": (OPEN, OPEN, MOVING, WALL, WALL, MOVING),
    "periodic_x": (PERIODIC, PERIODIC, WALL, WALL, MOVING, PRESSURE),
    "periodic_z": (OPEN, PRESSURE, SHEAR, SHEAR, PERIODIC, PERIODIC),
    "inlet": (INLET, PRESSURE, WALL, SHEAR, WALL, OPEN),
}
# partial tiles of both axes, a single short tile, tall grids; more planes than four slots
SIZES = [(17, 9, 13), (33, 17, 7), (13, 40, 6), (3, 2, 21)]


def _mesh(size, ends):
    m = build_uniform_mesh(*(2.0 * k for k in size), 1.0, visc=0.1)
    shift = {"periodic_x": (2.0 * size[0], 0.0, 0.0), "periodic_z": (0.0, 0.0, 2.0 * size[2])}.get(ends)
    m.set_boundaries(dict(zip(SIDES, ENDS[ends])), periodic_translation=shift)
    return m


def _params(size):
    return StepParams(visc=0.1, delta_t=0.35, channel_diameter=2.0 * size[1], body_force=(1e-5 / 3, -1e-6 / 7, 1e-6 / 11),
                      ref_rho=1.0, max_velocity=0.01, rho0=1.0, visc_factor_initial=1.0, testcase=2, viscosity_period=0)


def _state(n_cells, seed):
    rng = np.random.default_rng(seed)
    return [rng.uniform(0.99, 1.01, n_cells)] + [rng.uniform(-0.01, 0.01, n_cells) for _ in range(3)]


def _run(mesh, params, state, monkeypatch, walk, steps=4, membranes=()):
    monkeypatch.delenv("LBFS_GRID_WALK", raising=False)
    monkeypatch.delenv("LBFS_SEPARATE_KERNELS", raising=False)
    if walk:
        monkeypatch.setenv("LBFS_GRID_WALK", str(walk))
    else:
        monkeypatch.setenv("LBFS_SEPARATE_KERNELS", "1")
    with GpuSolver(mesh, params, list(membranes)) as s:
        assert s.launches_per_step() == (2 if walk else 4) + (6 if membranes else 0)
        s.set_state(*state)
        s.step(steps, graph=True)
        assert s.status() == 0
        return list(s.state()) + [s.field(_abi.LBFS_FIELD_T1)], s.nodes() if membranes else None


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("ends", ENDS)
def test_walks_of_any_length(size, ends, monkeypatch):
    m, p = _mesh(size, ends), _params(size)
    state = _state(m.n_cells, 7)
    one = _run(m, p, state, monkeypatch, 1)[0]
    for walk in sorted({2, 3, 5, size[2]}):
        for a, b in zip(one, _run(m, p, state, monkeypatch, walk)[0]):
            assert np.array_equal(a, b), walk
    for a, b in zip(one, _run(m, p, state, monkeypatch, 0)[0]):
        assert rel_err(a, b) < FP64_RTOL


@pytest.mark.parametrize("walk", [2, 5, 11])
def test_walks_of_two_instances(walk, monkeypatch):
    sizes, kinds = ((11, 9, 12), (18, 7, 10)), ("walls", "inlet")
    meshes = [_mesh(n, k) for n, k in zip(sizes, kinds)]
    e, p = concatenate(meshes), _params(sizes[0])
    states = [_state(m.n_cells, 11 + k) for k, m in enumerate(meshes)]
    got = _run(e, p, [np.concatenate(q) for q in zip(*states)], monkeypatch, walk)[0]
    for k, (m, st) in enumerate(zip(meshes, states)):
        for a, b in zip(got[:4], _run(m, p, st, monkeypatch, 1)[0]):
            assert np.array_equal(e.split(a)[k], b), k


def test_walks_across_an_interior_viscosity(monkeypatch):
    """A red cell whose interior has five times the viscosity (marked in the second step): the factors of the
    staged planes differ from plane to plane."""
    c = cases.shear_rbc(n=20, level=2, radius_cells=5.0, rotate=True)
    out = [_run(c.mesh, c.params, (c.rho, c.u, c.v, c.w), monkeypatch, w, 6, c.membranes) for w in (1, 2, 3, 7, 20, 0)]
    for state, nodes in out[1:-1]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0][0], state))
        assert np.array_equal(out[0][1], nodes)
    for a, b in zip(out[0][0], out[-1][0]):
        assert rel_err(a, b) < FP64_RTOL
    assert rel_err(out[0][1], out[-1][1]) < FP64_RTOL
