"""Workloads of the LBFS-IBM time step as a program that uses this framework runs them: fluid alone
and with red cells, FP64 and FP32 bulk, every kind of mesh, the loop on the host and on the device,
single handles, batched ensembles and the discrete adjoint.

A case is a dict of plain values; prepare() builds the host arrays from a seed and creates the handle
(mesh, membranes, initial state) that a simulation keeps, run() advances it by one output interval and
reads what such a program reads: the state records and accumulators into a device buffer, the node
positions, or the whole state through host arrays, or the adjoint's gradients.
"""
import math
import os
import sys
import tempfile
from dataclasses import replace

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "lbfs-ibm-ade-sp_b200"))
from lbfs_b200 import GpuSolver, _abi, cases  # noqa: E402

PRECISION = {"fp64": _abi.LBFS_FP64, "fp32": _abi.LBFS_FP32_BULK}
STENCIL = {"hat2": _abi.LBFS_IBM_HAT2, "peskin4": _abi.LBFS_IBM_PESKIN4, "vandermonde4": _abi.LBFS_IBM_VANDERMONDE4}


def _duct(name, nx, ny, nz, steps, precision="fp64", periodic=False, jitter=0.0, loop="host"):
    return dict(name=name, kind="duct", nx=nx, ny=ny, nz=nz, steps=steps, precision=precision, periodic=periodic,
                jitter=jitter, loop=loop)


def _shear(name, nx, ny, nz, steps, level, radius, precision="fp64", stencil="peskin4", mesh="uniform"):
    return dict(name=name, kind="shear", nx=nx, ny=ny, nz=nz, steps=steps, level=level, radius=radius,
                precision=precision, stencil=stencil, mesh=mesh)


def _channel(name, n, cells, radius, steps, precision):
    return dict(name=name, kind="channel", n=n, cells=cells, radius=radius, steps=steps, precision=precision)


def _ensemble(name, instances, low, high, steps, precision):
    return dict(name=name, kind="ensemble", instances=instances, low=low, high=high, steps=steps, precision=precision)


def _imported(name, n, radius, steps, time_stepping="local"):
    return dict(name=name, kind="imported", n=n, radius=radius, steps=steps, time_stepping=time_stepping)


def _adjoint(name, n, level, radius, steps, every):
    return dict(name=name, kind="adjoint", n=n, level=level, radius=radius, steps=steps, every=every)


def listed():
    return [
        # the smallest call: a driver that takes one step of a small duct at a time (the drop-in test's size)
        _duct("duct_12_single_step", 12, 12, 12, 1),
        # the reference's own use of its solver on its 32^3 duct: the state in from host arrays, its loop
        # with the convergence test (on the device), the state back to the host
        _duct("duct_32_device_loop", 32, 32, 32, 50, loop="device"),
        # a periodic channel of odd, unequal sizes in the FP32-bulk form
        _duct("duct_periodic_57x45x33_fp32", 57, 45, 33, 10, precision="fp32", periodic=True),
        # an odd-sized box with a small red cell on the reference's 2-point stencil
        _shear("shear_45x37x29_hat2", 45, 37, 29, 10, 2, 5.0, stencil="hat2"),
        # the single red cell in shear, the framework's main workload, in both precisions
        _shear("shear_64", 64, 64, 64, 10, 3, 8.0),
        _shear("shear_64_fp32", 64, 64, 64, 10, 3, 8.0, precision="fp32"),
        # the same flow larger than the L2 cache
        _shear("shear_128", 128, 128, 128, 10, 3, 12.0),
        # general-normal faces: red cells in a duct of jittered hexahedra, in both precisions, the larger
        # one the precision study's mesh
        _channel("jittered_72", 72, 4, 6.0, 10, "fp64"),
        _channel("jittered_128_fp32", 128, 16, 6.0, 10, "fp32"),
        # a batched parameter study: channels of different sizes with one to eight red cells each
        _ensemble("ensemble_12_fp32", 12, 16, 48, 10, "fp32"),
        # an imported OpenFOAM mesh with a red cell, every cell advanced with its own time step
        _imported("imported_40_local_dt", 40, 5.0, 10),
        # the gradient of a red cell's deformation through a window of steps
        _adjoint("adjoint_48", 48, 4, 8.0, 50, 25),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("duct", "duct", "shear", "shear", "channel", "ensemble", "imported", "adjoint"))
    precision = rng.choice(("fp64", "fp32"))
    if kind == "duct":
        loop = rng.choice(("host", "host", "device"))
        jitter = rng.choice((0.0, 0.0, 0.1))
        c = _duct("", log(10, 110), log(10, 110), log(10, 110), rng.choice((1, 5, 10)), precision,
                  rng.random() < 0.3 and jitter == 0.0, jitter, loop)
    elif kind == "shear":
        ny, nz = log(24, 110), log(24, 110)
        mesh = rng.choice(("uniform", "uniform", "uniform", "plateau"))
        stencil = "vandermonde4" if mesh == "plateau" else rng.choice(("hat2", "peskin4"))
        c = _shear("", log(24, 110), ny, nz, rng.choice((5, 10)), rng.choice((2, 3)),
                   round(rng.uniform(3.0, min(ny, nz, 64) / 8.0 + 1.0), 2), precision, stencil, mesh)
    elif kind == "channel":
        c = _channel("", log(32, 100), rng.randint(1, 4), round(rng.uniform(3.0, 6.0), 2), rng.choice((5, 10)), precision)
    elif kind == "ensemble":
        c = _ensemble("", rng.randint(2, 8), 16, rng.randint(20, 48), rng.choice((5, 10)), precision)
    elif kind == "imported":
        c = _imported("", log(20, 44), round(rng.uniform(2.5, 4.0), 2), rng.choice((5, 10)), rng.choice(("local", "min", "constant")))
    else:
        steps = rng.choice((20, 50))
        c = _adjoint("", log(28, 52), rng.choice((2, 3, 4)), round(rng.uniform(4.0, 6.0), 2), steps, steps // 2)
    del c["name"]
    return c


def _noise(case, seed, amplitude=1e-5):
    """Seeded perturbation of the velocity (the meshes and membranes of an ensemble do not follow the seed)."""
    rng = np.random.default_rng(seed)
    return replace(case, **{k: getattr(case, k) + rng.uniform(-amplitude, amplitude, case.mesh.n_cells) for k in "uvw"})


def _case(c, seed):
    """The host-side description of a case: mesh, parameters, membranes, initial state."""
    kind, prec = c["kind"], PRECISION[c.get("precision", "fp64")]
    if kind == "duct":
        return cases.poiseuille(c["nx"], ny=c["ny"], nz=c["nz"], seed=seed, precision=prec, periodic_x=c["periodic"],
                                jitter=c["jitter"], mesh_seed=seed)
    if kind == "shear":
        plateau = dict(mesh_type=4, plateau=(5.0, 0.3)) if c["mesh"] == "plateau" else {}
        return cases.shear_rbc(c["nx"], c["level"], c["radius"], u_wall=0.002, seed=seed, precision=prec,
                               ibm_stencil=STENCIL[c["stencil"]], n_cells_y=c["ny"], n_cells_z=c["nz"], rotate=True,
                               **plateau)
    if kind == "channel":
        return cases.jittered_channel(c["n"], c["cells"], radius_cells=c["radius"], seed=seed, precision=prec)
    if kind == "ensemble":
        return _noise(cases.ensemble(c["instances"], n_range=(c["low"], c["high"]), precision=prec), seed)
    if kind == "imported":
        # the importer sets no delta_h for the interior-viscosity update to go by: left out, as in the tests
        k = cases.shear_rbc(c["n"], 2, c["radius"], u_wall=0.002, seed=seed, rotate=True)
        stepping = {"local": _abi.LBFS_DT_LOCAL, "min": _abi.LBFS_DT_MIN, "constant": _abi.LBFS_DT_CONSTANT}
        k.params = replace(k.params, time_stepping=stepping[c["time_stepping"]], viscosity_period=0)
        with tempfile.TemporaryDirectory() as d:
            return cases.imported(k, d, jitter=0.05, seed=seed)
    k = cases.shear_rbc(c["n"], c["level"], c["radius"], u_wall=0.002, seed=seed, rotate=True)
    k.membranes = [replace(m, internal_viscosity_ratio=1.0) for m in k.membranes]
    return k


def prepare(c, seed):
    case = _case(c, seed)
    s = GpuSolver(case.mesh, case.params, case.membranes)
    s.set_state(case.rho, case.u, case.v, case.w)
    n = case.mesh.n_cells
    real = torch.float32 if case.params.precision == _abi.LBFS_FP32_BULK else torch.float64
    buf = torch.empty(s.halo_bytes(n), dtype=torch.uint8, device="cuda")
    cut = 4 * n * (4 if real is torch.float32 else 8)
    views = (buf[:cut].view(real).view(n, 4), buf[cut:].view(torch.float64).view(n, 4))
    return dict(case=c, solver=s, state=(case.rho, case.u, case.v, case.w), n=n, buf=buf, views=views)


def run(st):
    c, s = st["case"], st["solver"]
    if c.get("loop") == "device":
        s.set_state(*st["state"])
        done, residuals = s.step_until(c["steps"], 0.0)
        return {"steps": done, "residuals": residuals, "state": s.state()}
    if c["kind"] == "adjoint":
        J, grad, _ = s.adjoint(c["steps"], c["every"], membrane=0)
        s.halo_pack(0, st["n"], st["buf"].data_ptr())
        return {"J": J, "grad": grad, "state": st["views"], "nodes": s.nodes()}
    s.step(c["steps"], graph=True)
    s.halo_pack(0, st["n"], st["buf"].data_ptr())
    out = {"state": st["views"]}
    if s.total_nodes:
        out["nodes"] = s.nodes()
    return out


def _cells(c):
    if c["kind"] in ("duct", "shear"):
        return c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "ensemble":
        return sum(sp["n"] ** 3 for sp in cases.ensemble_specs(c["instances"], n_range=(c["low"], c["high"])))
    return c["n"] ** 3


def work(c):
    """Per step and cell: state and FP64 accumulator in and out; the face geometry (area, dt, normal, two
    offsets) and least-squares weights of a mesh that has them; about 60 operations for the gradients and
    60 for the update, and per face about 300 (axis-aligned) or 500 (general normal) for the 15
    reconstructed populations and the flux.  The adjoint's reverse step reads the stored gradients too
    and costs about three forward steps' operations."""
    real = 4 if c.get("precision") == "fp32" else 8
    general = c["kind"] in ("channel", "imported") or c.get("jitter", 0.0) > 0
    cells = _cells(c)
    per_cell = 2 * (4 * real + 32) + ((3 * 11 + 18) * real if general else 0)
    flops = 120 + 3 * (500 if general else 300)
    if c["kind"] == "adjoint":
        per_cell, flops = 3 * per_cell + 24 * real, 4 * flops
    return {"bytes": float(cells * per_cell * c["steps"]), "flops": float(cells * flops * c["steps"])}


# ---- the same steps in plain FP64 torch (fluid without membranes) -------------------------------

E = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 1), (-1, -1, -1),
              (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1), (-1, 1, 1), (1, -1, -1)], dtype=np.float64)
W = np.array([2.0 / 9.0] + [1.0 / 9.0] * 6 + [1.0 / 72.0] * 8)


def _equilibrium(s):
    """Equilibrium populations [.., 15] of states [.., 15 or 1, 4] (rho, u, v, w)."""
    e, w = torch.tensor(E, device=s.device), torch.tensor(W, device=s.device)
    eu = (e * s[..., 1:]).sum(-1)
    return w * s[..., 0] * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * (s[..., 1:] ** 2).sum(-1))


def _flux(nodes, tau, area, normal):
    """Flux (rho, u, v, w) through faces from the states at their 15 lattice nodes [f, 15, 4]."""
    e = torch.tensor(E, device=nodes.device)
    f = _equilibrium(nodes)
    rho, m = f.sum(-1), f @ e
    eq = _equilibrium(torch.cat([rho[:, None], m / rho[:, None]], 1)[:, None, :])
    f = eq - tau * (eq - f)
    en = (e * normal[:, None, :]).sum(-1) * f
    return torch.cat([en.sum(-1, keepdim=True), en @ e], 1) * area[:, None]


def exact(c, seed):
    if c["kind"] != "duct":
        return None
    k = _case(c, seed)
    m, p = k.mesh, k.params
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def on(a, *shape):
        t = torch.as_tensor(np.ascontiguousarray(a), device=dev)
        return t.reshape(shape) if shape else t

    nc, ni, nf, nb = m.n_cells, m.n_interior, m.n_faces, m.n_bc
    owner, neighbour = on(m.owner).long(), on(m.neighbour).long()
    stencil, lhs, rhs = on(m.gradient_stencil, nc, 6).long(), on(m.lhs_inverse, nc, 3, 3), on(m.rhs, nc, 6, 3)
    cen, fcen, normal = on(m.cell_centroid, -1, 3), on(m.face_centroid, nf, 3), on(m.face_normal, nf, 3)
    area, dt, vol = on(m.face_area), on(m.streaming_dt), on(m.cell_volume)[:nc]
    rt, vt, bc = on(m.bc_rho_type), on(m.bc_vel_type), on(m.bc_values, nb, 4)[:, [3, 0, 1, 2]]
    partner = on(m.periodic_node).long() if m.periodic_node is not None else None
    own_b = owner[ni:]
    types = torch.stack([rt, vt, vt, vt], 1)
    t1 = cen[owner] - fcen
    t2 = cen[neighbour] - fcen
    e = torch.tensor(E, device=dev)
    en = normal @ e.T                                   # [nf, 15]
    tau = p.visc * 3 / dt * p.gamma_inv
    force = on(np.array([0.0, *p.body_force]))
    s = on(np.stack([k.rho, k.u, k.v, k.w], 1))
    acc = s.clone()                                     # the accumulator starts from the primitive state

    def faces(a, b, full):
        """Flux through faces [a, b)."""
        o, n, d = owner[a:b], neighbour[a:b], dt[a:b]
        g1, g2 = grad[o], grad[n]
        at = lambda base, g, t: base - (g * t[:, None, :]).sum(-1)  # noqa: E731
        pi, pn = at(full[o], g1, t1[a:b]), at(full[n], g2, t2[a:b])
        p0, side = (pi + pn) * 0.5, en[a:b]
        if a == ni:                                     # boundary faces; the first ghost's is interior-like
            wall = torch.where(types == 1, bc, at(full[o], g2, t1[a:b]))
            edge = (n > nc)[:, None]
            p0 = torch.where(edge, wall, p0)
            pi, pn = torch.where(edge, p0, pi), torch.where(edge, p0, pn)
            g1 = torch.where(edge[..., None], g2, g1)
        gm = (g1 + g2) * 0.5
        if m.axis_aligned and a < ni:                   # weighted by the distances to the face
            x = (normal[a:b].abs() * (cen[n] - cen[o])).sum(-1)
            wa = ((normal[a:b].abs() * t2[a:b]).sum(-1) / x).abs()[:, None, None]
            wb = ((normal[a:b].abs() * t1[a:b]).sum(-1) / x).abs()[:, None, None]
            gm = g1 * wa + g2 * wb
        up, down = side > 0.001 * d[:, None], side < -0.001 * d[:, None]
        up, down = up[..., None], down[..., None]

        def reach(base, g):
            return base[:, None, :] - torch.einsum("fmx,kx->fkm", g, e) * d[:, None, None]

        nodes = torch.where(up, reach(pi, g1), torch.where(down, reach(pn, g2), reach(p0, gm)))
        return _flux(nodes, tau[a:b, None], area[a:b], normal[a:b])

    for _ in range(c["steps"]):
        own = s[own_b]
        other = s[partner] if partner is not None else own
        ghost = torch.where(types == 1, 2 * bc - own, torch.where(types == 3, other, own))
        full = torch.cat([s, ghost])
        d = full[stencil] - s[:, None, :]
        gi = torch.einsum("cij,cqj,cqm->cmi", lhs, rhs, d)
        r = cen[nc:] - cen[own_b]
        r2 = (r * r).sum(-1)
        gw = ((ghost - own) / r2[:, None])[..., None] * r[:, None, :]
        gb = torch.where((types == 1)[..., None], gw, gi[own_b] * (1 - normal[ni:].abs())[:, None, :])
        if partner is not None:
            gb = torch.where((types == 3)[..., None], gi[partner], gb)
        grad = torch.cat([gi, gb])
        res = torch.zeros_like(s)
        for a, b in [(x, min(x + 400000, ni)) for x in range(0, ni, 400000)] + [(ni, nf)]:
            flux = faces(a, b, full)
            res.index_add_(0, owner[a:b], -flux / vol[owner[a:b], None])
            if a < ni:
                res.index_add_(0, neighbour[a:b], flux / vol[neighbour[a:b], None])
        res = res + force
        acc = acc + p.delta_t * res
        s = torch.cat([acc[:, :1], acc[:, 1:] / acc[:, :1]], 1)
    if c["loop"] == "device":
        rms = res.square().mean(0).sqrt() / on(np.array([p.ref_rho] + [p.ref_rho * p.max_velocity] * 3))
        return {"steps": c["steps"], "residuals": rms, "state": tuple(s[:, q] for q in range(4))}
    rho0 = p.rho0 if c["precision"] == "fp32" else 0.0
    shift = on(np.array([0.0, 0.0, 0.0, rho0]))
    return {"state": (s[:, [1, 2, 3, 0]] - shift, acc[:, [1, 2, 3, 0]])}
