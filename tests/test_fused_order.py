"""The order of a cell's sums on uniform FP64 grids does not depend on how the fused pass cuts its tiles.

The pass walks tiles of columns over some planes; how long the walks are follows from all instances of a
handle together.  A cell whose upper neighbour lies in another walk takes that face's flux in the update
instead of inside the walk.  An instance of an ensemble and a slab of a mesh must evolve bit for bit as
they do in a handle of their own, so both places keep one order of sums.  The sizes are walked over
different lengths by the handles compared (more than one plane each), and at spacing 1.5 the ratio of
area and volume is no power of two, so that another place of the scaling shows in the last bits.
"""
import numpy as np
import pytest

from lbfs_b200 import GpuSolver, StepParams, _abi, build_uniform_mesh
from lbfs_b200.ensemble import concatenate
from lbfs_b200.slabs import SlabSolver, build_slab_mesh, slab_bounds, step_local

pytestmark = pytest.mark.gpu

WALL, OPEN = (2, 1, 1.0, 0.0, 0.0, 0.0), (2, 2, 1.0, 0.0, 0.0, 0.0)
MOVING = (2, 1, 1.0, 0.01, 0.002, -0.003)
BCS = {"left": OPEN, "right": OPEN, "bottom": WALL, "top": MOVING, "back": WALL, "front": MOVING}
# a force that does not fit in few bits, so that sums of the same terms in another order differ
PARAMS = StepParams(visc=0.1, delta_t=0.35, channel_diameter=64.0, body_force=(1e-5 / 3, -1e-6 / 7, 1e-6 / 11),
                    ref_rho=1.0, max_velocity=0.01, rho0=1.0, visc_factor_initial=1.0, testcase=2, viscosity_period=0)


def _box(n, spacing):
    m = build_uniform_mesh(*(spacing * k for k in n), 0.5 * spacing, visc=PARAMS.visc)
    m.set_boundaries(BCS)
    return m


def _state(n_cells, seed):
    rng = np.random.default_rng(seed)
    return [rng.uniform(0.99, 1.01, n_cells)] + [rng.uniform(-0.01, 0.01, n_cells) for _ in range(3)]


def _run(mesh, state, steps=4):
    with GpuSolver(mesh, PARAMS) as s:
        s.set_state(*state)
        s.step(steps, graph=True)
        assert s.launches_per_step() == 2  # the fused pass and the update
        assert s.status() == 0
        return s.state()


@pytest.mark.parametrize("spacing", [2.0, 1.5])
@pytest.mark.parametrize("sizes", [((40, 40, 40), (44, 44, 44)), ((48, 47, 45), (40, 41, 66), (63, 50, 49))],
                         ids=["40_44", "three"])
def test_instances_equal_handles_of_their_own(sizes, spacing):
    meshes = [_box(n, spacing) for n in sizes]
    states = [_state(m.n_cells, 5 + k) for k, m in enumerate(meshes)]
    e = concatenate(meshes)
    got = _run(e, [np.concatenate(q) for q in zip(*states)])
    for k, (m, st) in enumerate(zip(meshes, states)):
        for a, b in zip(got, _run(m, st)):
            assert np.array_equal(e.split(a)[k], b), k


@pytest.mark.parametrize("spacing", [2.0, 1.5])
def test_slabs_equal_the_whole_mesh(spacing):
    n, nz = 64, 128
    mesh = _box((n, n, nz), spacing)
    state = _state(mesh.n_cells, 3)
    want = _run(mesh, state)
    bounds = slab_bounds(nz, 2)
    slabs = []
    for r in range(2):
        slab = build_slab_mesh(n * spacing, n * spacing, nz * spacing, 0.5 * spacing, bounds, r, bcs=BCS, visc=PARAMS.visc)
        slabs.append(SlabSolver(slab, PARAMS))
        slabs[-1].set_state(*state)
    step_local(slabs, 4, "cuda:0")
    for s, (z0, z1) in zip(slabs, bounds):
        for a, b in zip(s.owned_state(), want):
            assert np.array_equal(a, b[z0 * n * n:z1 * n * n])
        s.solver.close()


def _plateau(n):
    m = build_uniform_mesh(*(2.0 * k for k in n), 1.0, visc=PARAMS.visc, mesh_type=4, plateau_width=5.0, plateau_slope=0.3)
    m.set_boundaries(BCS)
    return m


@pytest.mark.parametrize("kinds", ["2 1.5", "1.5 2 1", "p 2", "2 p 1.5 p", "p 1.5 p"])
def test_instances_of_different_meshes_equal_handles_of_their_own(kinds):
    """Grids of different spacings and rectilinear ones (p) in one handle: each instance takes the kernels,
    and the constants, that it takes alone; the gradient, flux and ghost fields too."""
    meshes = [_plateau((14 + k, 12, 10)) if s == "p" else _box((13, 17 + k, 12), float(s)) for k, s in enumerate(kinds.split())]
    states = [_state(m.n_cells, 20 + k) for k, m in enumerate(meshes)]
    e = concatenate(meshes)

    def run(mesh, state):
        with GpuSolver(mesh, PARAMS) as s:
            s.set_state(*state)
            s.step(3, graph=True)
            s.step(2)
            s.keep_residuals(True)
            s.step(1)
            assert s.status() == 0
            return s.state(), s.field(_abi.LBFS_FIELD_RESIDUAL).reshape(-1, 4), \
                s.field(_abi.LBFS_FIELD_GRADIENTS).reshape(-1, 12), s.field(_abi.LBFS_FIELD_GHOST).reshape(-1, 4)

    state, res, grad, ghost = run(e, [np.concatenate(q) for q in zip(*states)])
    b0 = 0
    for k, (m, st) in enumerate(zip(meshes, states)):
        own = run(m, st)
        for a, b in zip(state, own[0]):
            assert np.array_equal(e.split(a)[k], b), k
        assert np.array_equal(e.split(res)[k], own[1]), k
        assert np.array_equal(e.split(grad)[k], own[2][:m.n_cells]), k
        assert np.array_equal(ghost[b0:b0 + m.n_bc], own[3]), k
        assert np.array_equal(grad[e.n_cells + b0:e.n_cells + b0 + m.n_bc], own[2][m.n_cells:]), k
        b0 += m.n_bc


def test_a_mixed_handle_through_the_other_entry_points(monkeypatch):
    """Uniform grids of two spacings and a rectilinear one in a handle: the device loop, eager steps, several
    steps a graph, a restore and tuning leave the states of single graph steps; the adjoint is that of a
    handle on the separate kernels (which it records with)."""
    meshes = [_box((13, 17, 12), 2.0), _plateau((14, 12, 10)), _box((12, 11, 15), 1.5)]
    e = concatenate(meshes)
    state = [np.concatenate(q) for q in zip(*(_state(m.n_cells, 40 + k) for k, m in enumerate(meshes)))]

    def handle():
        s = GpuSolver(e, PARAMS)
        s.set_state(*state)
        assert s.launches_per_step() == 5  # the pass, three kernels beside it, the update
        return s

    def same(s, t):
        return all(np.array_equal(a, b) for a, b in zip(s.state(), t.state()))

    with handle() as ref, handle() as s, handle() as t:
        for _ in range(6):
            ref.step(1, graph=True)
        assert s.step_until(6, 0.0)[0] == 6 and same(s, ref)
        t.step(3)
        blob = t.checkpoint()
        t.step(9, graph=True)
        t.autotune(reps=3)
        t.restore(blob)
        t.step(3, graph=True)
        assert same(t, ref)
        for _ in range(300):
            s.step(2, graph=True)
        for _ in range(600):
            ref.step(1, graph=True)
        assert same(s, ref) and s.status() == 0
    weights = np.random.default_rng(2).uniform(-1, 1, 3 * e.n_cells)
    out = []
    for separate in (False, True):
        if separate:
            monkeypatch.setenv("LBFS_SEPARATE_KERNELS", "1")
        with GpuSolver(e, PARAMS) as s:
            s.set_state(*state)
            J, grad, _ = s.adjoint(8, 4, weights=weights)
            out.append((J, grad, s.state(), s.field(_abi.LBFS_FIELD_GRADIENTS)))
    assert out[0][:2] == out[1][:2]
    assert all(np.array_equal(a, b) for a, b in zip(out[0][2], out[1][2])) and np.array_equal(out[0][3], out[1][3])
