"""The fused fluid step of uniform grids against the separate kernels.

On uniform meshes a step forms the face fluxes and cell sums in one kernel over tiles of columns
(lbfs_fused.cu); LBFS_SEPARATE_KERNELS keeps a handle on the gradient, face and update kernels.  The
two evaluate the same formulas with other roundings (closed forms of the corner sums, one product per
difference), so FP64 states agree to the parity bound.
"""
import numpy as np
import pytest

from helpers import FP64_RTOL, rel_err


def _handle(c, monkeypatch, separate):
    from lbfs_b200 import GpuSolver
    if separate:
        monkeypatch.setenv("LBFS_SEPARATE_KERNELS", "1")
    else:
        monkeypatch.delenv("LBFS_SEPARATE_KERNELS", raising=False)
    s = GpuSolver(c.mesh, c.params, c.membranes)
    s.set_state(c.rho, c.u, c.v, c.w)
    return s


def _duct(nx, ny, nz, precision=0, periodic=False, inlet=False):
    from lbfs_b200 import cases
    c = cases.poiseuille(nx, ny=ny, nz=nz, precision=precision, periodic_x=periodic)
    if inlet:  # the square-duct inlet profile (type 9) and a Dirichlet density outlet: no zero-gradient x end
        c.bcs = dict(c.bcs, left=(2, 9, 1.0, 1e-5, 0.0, 0.0), right=(1, 2, 1.0, 0.0, 0.0, 0.0))
        c.mesh.set_boundaries(c.bcs)
    return c


# two cells thick axes (the generator's least); one column, one row and one plane beyond a tile of 16 x 8 (13 = 7 + 6 and 5 x 3 - 2
# splits); more planes than a walk; a row longer than a block
SIZES = [(2, 5, 3), (2, 2, 7), (17, 9, 5), (13, 13, 4), (33, 17, 6), (150, 3, 3), (3, 130, 2), (16, 8, 70)]


@pytest.mark.gpu
@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
@pytest.mark.parametrize("ends", ["open", "periodic", "inlet"])
def test_fused_step_equals_separate_kernels(size, ends, monkeypatch):
    from lbfs_b200 import _abi
    out = []
    for separate in (False, True):
        c = _duct(*size, periodic=ends == "periodic", inlet=ends == "inlet")
        s = _handle(c, monkeypatch, separate)
        assert s.launches_per_step() == (4 if separate else 2)
        s.keep_residuals(True)
        s.step(2)
        s.step(3, graph=True)
        out.append(dict(grad=s.field(_abi.LBFS_FIELD_GRADIENTS), flux=s.field(_abi.LBFS_FIELD_FACE_FLUX),
                        ghost=s.field(_abi.LBFS_FIELD_GHOST), t1=s.field(_abi.LBFS_FIELD_T1),
                        res=s.field(_abi.LBFS_FIELD_RESIDUAL).reshape(-1, 4), rms=s.residuals(),
                        state=np.array(s.state())))
        assert s.status() == 0
        s.close()
    a, b = out
    for key in ("grad", "flux", "ghost", "t1"):
        assert rel_err(a[key], b[key]) < FP64_RTOL, key
    for q in range(4):
        # sums of six fluxes of the pressure's size (area / 3 / volume = 1/6) that cancel: rounding of that size
        assert np.max(np.abs(a["res"][:, q] - b["res"][:, q])) < 1e-15 * 10
        if np.any(b["state"][q]):
            assert rel_err(a["state"][q], b["state"][q]) < FP64_RTOL, q
    assert np.allclose(a["rms"], b["rms"], rtol=1e-8, atol=1e-13)


@pytest.mark.gpu
def test_fields_of_the_last_step_are_kept(monkeypatch):
    """The gradient, flux and ghost fields are formed on request from the state the last step started
    from: a new state, a restore, or asking twice does not change them."""
    from lbfs_b200 import _abi, cases
    c = cases.shear_rbc(n=16, level=2, radius_cells=3.0)
    s = _handle(c, monkeypatch, False)
    which = (_abi.LBFS_FIELD_GRADIENTS, _abi.LBFS_FIELD_FACE_FLUX, _abi.LBFS_FIELD_GHOST)
    s.step(3, graph=True)
    blob = s.checkpoint()
    first = [s.field(w) for w in which]
    s.set_state(c.rho, c.u, c.v, c.w)
    assert all(np.array_equal(a, s.field(w)) for a, w in zip(first, which))
    s.step(2, graph=True)
    moved = [s.field(w) for w in which]
    assert not any(np.array_equal(a, b) for a, b in zip(first, moved))
    s.restore(blob)
    s.step(1, graph=True)
    t = _handle(c, monkeypatch, False)
    t.step(4, graph=True)
    assert all(np.array_equal(s.field(w), t.field(w)) for w in which)
    s.close()
    t.close()


@pytest.mark.gpu
def test_device_memory_of_a_handle(monkeypatch):
    """What the fused step keeps beside the separate kernels' arrays is the state the last step started
    from and the cell sums (64 B a cell) and its tables; and a uniform mesh's weights, inverses and face
    geometry, which the kernels take from their parameters, are not uploaded: some 450 B a cell by the
    arrays' sizes (state and accumulator 64, gradients and fluxes 192, stencil and faces 72, volumes,
    viscosity, centroids and codes 52, kept state and sums 64, and boundary tables)."""
    import torch
    from lbfs_b200 import cases
    torch.cuda.init()
    c = cases.poiseuille(96)
    held = {}
    for separate in (False, True):
        _handle(c, monkeypatch, separate).close()  # the library's own contexts and modules
        free = torch.cuda.mem_get_info()[0]
        s = _handle(c, monkeypatch, separate)
        held[separate] = (free - torch.cuda.mem_get_info()[0]) / c.mesh.n_cells
        s.close()
    assert held[False] < held[True] + 90, held
    assert held[False] < 660, held  # allocations are rounded up to 2 MB, some 40 of them: 95 B a cell
