"""The separate gradient, face and update kernels where the fused step would stand in for them.

FP64 handles of uniform meshes take the fused step, whose launches the gradient and flux block sizes, the
chunks of the two-stream pipeline and the coded geometry do not touch.  Rectilinear FP64 meshes, FP32
handles and the adjoint take the separate kernels; here they run on uniform meshes, FP64 (with
LBFS_SEPARATE_KERNELS) and FP32, and the launch counts show that they did.
"""
import numpy as np
import pytest

from lbfs_b200 import GpuSolver, _abi, cases

pytestmark = [pytest.mark.gpu, pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])]


@pytest.fixture(autouse=True)
def _separate(monkeypatch):
    monkeypatch.setenv("LBFS_SEPARATE_KERNELS", "1")


def _handle(c, launches, **shape):
    s = GpuSolver(c.mesh, c.params, c.membranes)
    s.set_launch_shape(**shape)
    s.set_state(c.rho, c.u, c.v, c.w)
    assert s.launches_per_step() == launches
    return s


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def test_pipelined_gradients_and_fluxes(precision):
    """flux_chunks K: K gradient and K face launches on two streams, the same fields bit for bit."""
    c = cases.shear_rbc(n=40, level=3, radius_cells=6.0, precision=precision)
    out = []
    for k in (1, 2, 4, 8):
        with _handle(c, 2 * k + 2 + 6, flux_chunks=k) as s:
            s.keep_residuals(True)
            s.step(2)
            s.step(4, graph=True)
            assert s.status() == 0
            out.append((*s.state(), s.nodes(), s.field(_abi.LBFS_FIELD_GRADIENTS), s.field(_abi.LBFS_FIELD_FACE_FLUX),
                        s.field(_abi.LBFS_FIELD_RESIDUAL), s.residuals()))
    assert all(_same(out[0], o) for o in out[1:])


def test_launch_shapes(precision):
    """Block sizes of the gradient and flux kernels, with and without chunks."""
    c = cases.shear_rbc(n=24, level=2, radius_cells=4.0, precision=precision)
    shapes = [{}, dict(gradient_threads=256, flux_threads=64, general_flux_threads=256, flux_chunks=4),
              dict(gradient_threads=512, flux_threads=256, general_flux_threads=64),
              dict(gradient_threads=128, flux_threads=64, flux_chunks=2)]
    out = []
    for shape in shapes:
        with _handle(c, 2 * shape.get("flux_chunks", 1) + 2 + 6, **shape) as s:
            s.step(6, graph=True)
            out.append((*s.state(), s.nodes()))
    assert all(_same(out[0], o) for o in out[1:])


@pytest.mark.parametrize("cluster,chunks", [(0, 1), (8, 1), (0, 4)])
def test_membranes_behind_the_gradient_launch(precision, cluster, chunks):
    c = cases.shear_rbc(n=32, level=2, radius_cells=5.0, precision=precision)
    out = []
    for after in (0, 1):
        with _handle(c, 2 * chunks + 2 + (3 if cluster else 6), membrane_after_k1=after, membrane_cluster=cluster,
                     flux_chunks=chunks) as s:
            s.step(3, graph=True)
            s.step(1)
            s.step(4, graph=True)
            assert s.status() == 0
            out.append((*s.state(), s.nodes(), s.residuals()))
    assert _same(*out)


def test_coded_geometry_equals_generic(precision, monkeypatch):
    c = cases.shear_rbc(n=16, level=2, radius_cells=3.0, precision=precision)
    out = []
    for generic in (False, True):
        if generic:
            monkeypatch.setenv("LBFS_GENERIC_GEOMETRY", "1")
        with _handle(c, 2 + 2 + 6) as s:
            s.step(6, graph=True)
            assert s.status() == 0
            out.append((*s.state(), s.nodes(), s.residuals(), s.field(_abi.LBFS_FIELD_GRADIENTS),
                        s.field(_abi.LBFS_FIELD_FACE_FLUX)))
    assert _same(*out)
