"""Performance cases of the two-phase residual-and-update engine.

Each case is a call, or a short run of calls, that a program built on this
library makes: inject a state, march some steps with diagnostics and read the
state back (the body of the reference's time loop between two restarts); step
a batch of small meshes as the server does; build the overset tables of a new
mesh; form the time step of a state that lives in the caller's own buffers.
Mesh families, physical parameters and sizes are those of
hydraphase.cases, the tests and bench.py.

Keys of a case: "kind"; the mesh as "a", "b", "c" (hexes per direction, 6
tetrahedra each; see _built); "precision"; "steps" per pass; "flux" (myflux);
"scheme" ("ref": the reference's four-stage scheme with viscous terms, "ssp":
SSP-RK3, K = 5); "layers" (FP64 wall layers of the mixed variant); "count"
(meshes of a batch).
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multiphase-code_b200"))
from hydraphase import PREC_FP64, PREC_FP64_PARITY, PREC_MIXED, Batch, Case, cases, lib  # noqa: E402
from hydraphase.engine import overset_build, overset_hole_cut  # noqa: E402

PRECISION = {"fp64_parity": PREC_FP64_PARITY, "fp64": PREC_FP64, "mixed": PREC_MIXED}


def _case(kind, a, b, c, precision="fp64_parity", steps=10, flux=2, scheme="ssp", layers=0, count=1, **more):
    return dict(kind=kind, a=a, b=b, c=c, precision=precision, steps=steps, flux=flux, scheme=scheme, layers=layers,
                count=count, **more)


def listed():
    return [
        # time step of a caller-owned state (48,000 tets), no handle: the smallest call there is
        _case("dt", 20, 20, 20, steps=1, name="dt_48k"),
        # a toy box of 2,058 tets, as a new user or a unit test marches it: launches and latency
        _case("bubble", 7, 7, 7, steps=20, name="bubble_2k_parity"),
        # the shock-bubble configuration at its stated size, in the reference's own scheme
        _case("bubble", 20, 20, 20, scheme="ref", name="bubble_48k_parity_ref"),
        # one case of the serving stream near its upper end, odd side
        _case("bubble", 31, 31, 31, precision="mixed", steps=20, name="bubble_179k_mixed"),
        # a batch of small serving cases of odd sizes in one handle
        _case("batch", 10, 11, 24, precision="mixed", steps=20, count=6, name="batch_6_mixed"),
        # viscous cylinder, reduced O-grid of the tests
        _case("cylinder", 40, 64, 8, name="cylinder_123k_parity"),
        # the cylinder on the O-grid that the profiles are taken on: FP64 parity,
        # mixed, and mixed with FP64 layers at the wall
        _case("cylinder", 80, 128, 16, steps=5, name="cylinder_983k_parity"),
        _case("cylinder", 80, 128, 16, precision="mixed", name="cylinder_983k_mixed"),
        _case("cylinder", 80, 128, 16, precision="mixed", layers=40, steps=5, name="cylinder_983k_mixed_walls"),
        # the precision-stress shock over a lattice of bubbles, its full size: the largest mesh
        _case("lattice", 60, 60, 90, precision="mixed", steps=5, name="lattice_1944k_mixed"),
        # overset cylinder with fringe interpolation, FP64 with FMA
        _case("overset", 60, 48, 5, precision="fp64", steps=5, name="overset_246k_fp64"),
        # hole cut and donor search of that mesh on the device, as after every regridding
        _case("tables", 60, 48, 5, steps=1, name="overset_tables_246k"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["dt", "bubble", "bubble", "bubble", "batch", "cylinder", "cylinder", "cylinder", "lattice",
                       "overset"])
    flux = rng.choice([2, 2, 2, 1])
    prec = rng.choice(["fp64_parity", "fp64_parity", "mixed", "mixed", "fp64"])
    if kind == "dt":
        n = round(_log(rng, 4, 60))
        return _case("dt", n, n + rng.randrange(3), n + rng.randrange(5), steps=1)
    if kind == "bubble":
        n = round(_log(rng, 4, 45))
        return _case("bubble", n, n + rng.randrange(3), n + rng.randrange(5), prec, steps=rng.randint(3, 12),
                     flux=flux, scheme=rng.choice(["ssp", "ssp", "ref"]))
    if kind == "batch":
        return _case("batch", rng.randint(5, 9), rng.randint(10, 13), rng.randint(14, 24),
                     rng.choice(["mixed", "fp64_parity"]), steps=rng.randint(5, 20), count=rng.randint(2, 9))
    if kind == "lattice":
        n = rng.randint(15, 50)
        return _case("lattice", n, n + rng.randrange(4), 3 * n // 2 + rng.randrange(4), prec, steps=rng.randint(2, 6))
    if kind == "overset":
        return _case("overset", rng.randint(36, 64), rng.randint(24, 56), rng.randint(3, 6), prec, steps=rng.randint(2, 6))
    f = _log(rng, 0.25, 1.0)
    a, b, c = round(72 * f) + rng.randrange(6), round(110 * f) + rng.randrange(9), round(13 * f) + rng.randrange(2)
    # (the central flux, without limiting, carries the smooth flow only)
    return _case("cylinder", a, b, c, prec, steps=rng.randint(2, 8), flux=rng.choice([flux, flux, 3]), scheme=rng.choice(["ssp", "ssp", "ref"]),
                 layers=rng.choice([0, 0, round(40 * f)]) if prec == "mixed" else 0)


# --- inputs -------------------------------------------------------------------
@functools.lru_cache(maxsize=3)
def _built(kind, a, b, c):
    """The mesh of a case with its base state: (CaseSpec, blocks of an overset
    mesh or None).  Kept per process, as a program keeps its mesh."""
    if kind in ("dt", "bubble"):
        return cases.shock_bubble_on(cases.box_mesh(a, b, c, jitter=0.1, seed=1, bc_type=5), alpha_min=0.1), None
    if kind == "cylinder":
        return cases.cylinder(nr=a, nt=b, nz=c, alpha_w_drop=1e-5, alpha_w_bg=1e-6), None
    if kind == "lattice":
        return cases.shock_lattice(nx=a, ny=b, nz=c), None
    ov = cases.overset_cylinder(bg=(a, a, c), comp=(b, 2 * b, c), box=((-6.0, -6.0, 0.0), (6.0, 6.0, 4.0)),
                                alpha_w_drop=1e-5, alpha_w_bg=1e-6)
    return ov.spec, ov.block


def _centroids(m):
    el = m.elem[:, :4] - 1
    return [(q[el[:, 0]] + q[el[:, 1]] + q[el[:, 2]] + q[el[:, 3]]) * 0.25 for q in (m.x, m.y, m.z)]


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t.numpy()


def _state(spec, kind, rng):
    """cu and ghost primitives of one seed: the base state with a smooth gust
    on both phases' velocities, the energies following; a box also moves its
    bubble, and its shock has another strength."""
    m, f = spec.mesh, spec.flow
    x = _centroids(m)
    if kind in ("dt", "bubble", "batch"):
        b = cases.Built(m, np.stack(x, axis=1), None)
        spec = cases.shock_bubble_on(b, radius=rng.uniform(0.1, 0.3), p_post=math.exp(rng.uniform(math.log(1e8), math.log(2e9))),
                                     center=tuple(rng.uniform(0.4, 0.6, 3)), alpha_min=0.1)
    cu = spec.cu.copy()
    scale = 2.0 if kind in ("cylinder", "overset") else 0.5
    for r in (0, 5):
        old = 0.5 * (cu[r + 1] ** 2 + cu[r + 2] ** 2 + cu[r + 3] ** 2) / cu[r]
        if r == 0:
            gust = []
            for k in range(3):
                w = rng.uniform(0.5, 2.0, 3)
                gust.append(scale * np.sin(w[0] * x[0] + w[1] * x[1] + w[2] * x[2] + rng.uniform(0, 6)))
        for k in range(3):
            cu[r + 1 + k] += cu[r] * gust[k]
        cu[r + 4] += 0.5 * (cu[r + 1] ** 2 + cu[r + 2] ** 2 + cu[r + 3] ** 2) / cu[r] - old
    return _pinned(cu), _pinned(cases.ghost_prims_from_parents(m, cu, f["gamag"], f["gamap"], f["pinf"]))


def _params(case, spec):
    # CFL: 0.05 for the shock boxes, 0.25 for the viscous cylinder, as bench.py runs them
    wet = case["kind"] in ("cylinder", "overset")
    over = dict(precision=PRECISION[case["precision"]], myflux=case["flux"], cfl=0.25 if wet else 0.05,
                wall_fp64_layers=case["layers"])
    if case["scheme"] == "ref":
        over.update(rk_scheme=0, venkat_k=0.3, inviscid=0)
    return spec.params(**over)


def _batch_specs(case):
    return [_built("bubble", n, n, n)[0] for n in
            np.unique(np.linspace(case["a"], case["c"], case["count"]).round().astype(int))]


def _overset(spec, block):
    """Mesh with the library's hole cut and fringe marks, and the donor table."""
    mesh = cases.MeshArrays(spec.mesh.x, spec.mesh.y, spec.mesh.z, spec.mesh.elem.copy(), spec.mesh.ghost)
    mesh.elem[:, 8] = 1
    mesh.elem[:, 8], _ = overset_hole_cut(mesh, block, wall_type=6, margin=0.7, device=True)
    mesh.elem[:, 8], table = overset_build(mesh, block, layers=2, outer_type=7, device=True)
    return mesh, table


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    st = {"kind": kind, "steps": case["steps"]}
    if kind == "batch":
        specs = _batch_specs(case)
        h = st["handle"] = Batch([s.mesh for s in specs], _params(case, specs[0]))
        for c, s in enumerate(specs):
            h.set_state(c, 0.0, *_state(s, kind, rng))
        return st
    spec, block = _built("overset" if kind == "tables" else kind, case["a"], case["b"], case["c"])
    if kind == "tables":
        # another mesh for every seed: the component's grid turned a little, as a moving body turns it
        m, t = spec.mesh, rng.uniform(0.0, 0.02)
        comp = np.unique(m.elem[block == 1, :4]) - 1
        x, y = m.x.copy(), m.y.copy()
        x[comp], y[comp] = (math.cos(t) * m.x[comp] - math.sin(t) * m.y[comp],
                            math.sin(t) * m.x[comp] + math.cos(t) * m.y[comp])
        elem = m.elem.copy()
        elem[:, 8] = 1
        st.update(mesh=cases.MeshArrays(x, y, m.z, elem, m.ghost), block=block)
        return st
    cu, gp = _state(spec, kind, rng)
    if kind == "dt":
        m = spec.mesh
        p = np.stack([m.x, m.y, m.z], axis=1)[m.elem[:, :4] - 1]
        dl = np.min([np.linalg.norm(p[:, i] - p[:, j], axis=1) for i in range(4) for j in range(i)], axis=0)
        st.update(cn=torch.from_numpy(cu).cuda(), dl=torch.from_numpy(dl).cuda(), params=_params(case, spec),
                  dt=torch.empty(1, dtype=torch.float64, device="cuda"))
        return st
    mesh, table = (spec.mesh, None) if kind != "overset" else _overset(spec, block)
    h = Case(mesh, _params(case, spec))
    if table is not None:
        h.set_overset(table)
    st.update(handle=h, cu=cu, gp=gp, out=(_pinned(np.empty_like(cu)), _pinned(np.empty((6, max(mesh.nghosts, 1))))))
    return st


# --- one pass -----------------------------------------------------------------
def run(st):
    kind = st["kind"]
    if kind == "dt":
        cn, dl = st["cn"], st["dl"]
        rc = lib().hp_dt_noalloc(cn.data_ptr(), cn.shape[1], dl.data_ptr(), cn.shape[1], ctypes.byref(st["params"]),
                                 st["dt"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError("hp_dt_noalloc: %d" % rc)
        return st["dt"]
    if kind == "tables":
        st["mesh"].elem[:, 8] = 1
        st["mesh"].elem[:, 8], holes = overset_hole_cut(st["mesh"], st["block"], wall_type=6, margin=0.7, device=True)
        iblank, t = overset_build(st["mesh"], st["block"], layers=2, outer_type=7, device=True)
        return {"iblank": iblank, "holes": holes, "fringe": t.fringe, "donor": t.donor, "weight": t.weight}
    h = st["handle"]
    if kind == "batch":
        # the cases of a batch go on from where the last pass left them
        diag = h.step(st["steps"])
        return [dict(_told(h.state(c)), **d) for c, d in enumerate(diag)]
    h.set_state(0.0, st["cu"], st["gp"])
    diag = h.step(st["steps"])
    return dict(_told(h.state(out=st["out"])), **diag)


def _told(state):
    return {"cu": state[1], "ghosts": state[2]}


# --- what a pass cannot do without --------------------------------------------
def _cells(case):
    if case["kind"] == "batch":
        return sum(s.mesh.neles for s in _batch_specs(case))
    a, b, c = case["a"], case["b"], case["c"]
    return 6 * (a * a * c + 2 * b * b * c if case["kind"] in ("overset", "tables") else a * b * c)


def work(case):
    n = _cells(case)
    if case["kind"] == "dt":
        return {"bytes": 88.0 * n, "flops": 90.0 * n}        # ten variables and the edge length; EOS recovery
    if case["kind"] == "tables":
        return {"bytes": 250.0 * n, "flops": 100.0 * n}      # nodes, faces and centroids once; one test per cell
    stages = 4 if case["scheme"] == "ref" else 3
    # bytes: per cell and stage the state, primitives, gradients, geometry and
    # right-hand-side terms once each (half of it in FP32 in the mixed
    # variant); flops: LSQ gradients and limiter 1,300, four faces 1,300,
    # sources, recovery and update 300 per stage; JST 300 and, where they
    # are on, viscous faces 2,800 per step
    stage_bytes = 566.0 if case["precision"] == "mixed" else 772.0
    step_flops = 2900.0 * stages + 300.0 + (2800.0 if case["kind"] in ("cylinder", "overset") or case["scheme"] == "ref" else 0.0)
    return {"bytes": n * (case["steps"] * stages * stage_bytes + 160.0), "flops": n * case["steps"] * step_flops}


# --- the same in 64 bits, in plain torch --------------------------------------
def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "tables":
        return None       # whole numbers, and the weights that belong to them
    if kind == "batch":
        specs = _batch_specs(case)
        states = [_state(s, kind, rng) for s in specs]
        p = _params(case, specs[0])
        return [_March(s.mesh, p).run(*x, case["steps"]) for s, x in zip(specs, states)]
    spec, block = _built(kind, case["a"], case["b"], case["c"])
    cu, gp = _state(spec, kind, rng)
    p = _params(case, spec)
    if kind == "dt":
        w = _March(spec.mesh, p)
        return (p.cfl * w.dtmin(w.recover(_dev(cu))[0])).reshape(1)
    mesh, table = (spec.mesh, None) if kind != "overset" else _overset(spec, block)
    return _March(mesh, p, table).run(cu, gp, case["steps"])


def _dev(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to("cuda" if torch.cuda.is_available() else "cpu", dtype)


UG, VG, WG, TG, PG, PP, AG, AP, UP, VP, WP, TP, RG, RP = range(14)
R_GAS, AMU_P, PR_P = 287.0, 0.001, 10.0
E6, E8 = float(np.float32(1e-6)), float(np.float32(1e-8))
C23 = float(np.float32(2.0) / np.float32(3.0))
GRAD = (UG, VG, WG, TG, UP, VP, WP, TP, PG, PP, AG, RG, RP)


def _det(a, b, c):
    """Determinant of the 3 x 3 matrix with columns a, b, c."""
    return (a[0] * (b[1] * c[2] - b[2] * c[1]) - a[1] * (b[0] * c[2] - b[2] * c[0]) + a[2] * (b[0] * c[1] - b[1] * c[0]))


def _solve(A, r):
    """Cramer's rule for the symmetric matrix with columns A."""
    d = _det(*A)
    return torch.stack([_det(r, A[1], A[2]) / d, _det(A[0], r, A[2]) / d, _det(A[0], A[1], r) / d])


def _normal(x, w):
    """Columns of sum_k x_k x_k^T / w_k over points x (3, k, n)."""
    return [(x * x[i] / w).sum(1) for i in range(3)]


class _March:
    """The explicit step on one mesh, (variables, cells) tensors in the
    mesh's own order, ghosts after the elements."""

    def __init__(self, mesh, p, table=None):
        self.p = p
        self.ne, self.ng = mesh.neles, mesh.nghosts
        el = _dev(mesh.elem, torch.int64)
        gh = _dev(mesh.ghost, torch.int64)
        self.par, self.gid, self.gtype = gh[:, 0] - 1, gh[:, 1] - 1, gh[:, 2]
        node, self.nc, self.blank = (el[:, :4] - 1).T, (el[:, 4:8] - 1).T, el[:, 8]
        xyz = _dev(np.stack([mesh.x, mesh.y, mesh.z]))
        q = xyz[:, node]                                                  # (3, 4, ne)
        of = [[1, 2, 3], [0, 2, 3], [0, 1, 3], [0, 1, 2]]                 # the nodes of face k, opposite node k
        fq = torch.stack([q[:, o] for o in of])                           # (face, 3, node, ne)
        s = 0.5 * torch.linalg.cross(fq[:, :, 1] - fq[:, :, 0], fq[:, :, 2] - fq[:, :, 0], dim=1)
        out = (s * (fq[:, :, 0] - q.transpose(0, 1))).sum(1, keepdim=True)
        self.sc = torch.where(out < 0, -s, s)                             # (face, 3, ne)
        self.vol = (torch.linalg.cross(q[:, 2] - q[:, 0], q[:, 3] - q[:, 0], dim=0) * (q[:, 1] - q[:, 0])).sum(0).abs() / 6
        self.dl = torch.stack([(q[:, i] - q[:, j]).square().sum(0).sqrt() for i in range(4) for j in range(i)]).amin(0)
        self.fch, self.fcv = fq.sum(2) * 0.3333, fq.mean(2)
        xc = q.mean(1)
        side = gh[:, 3] - 1
        self.xc = torch.zeros(3, self.ne + self.ng, dtype=xc.dtype, device=xc.device)
        self.xc[:, :self.ne] = xc
        self.xc[:, self.gid] = 2 * self.fcv[side, :, self.par].T - xc[:, self.par]
        zc, zn = xc[2, self.par], xyz[2]
        self.dd = torch.where(zc > float(np.float32(0.1)), zn.max() - zc, zc - zn.min()).abs()
        typ = torch.zeros(self.ne + self.ng, dtype=torch.int64, device=xc.device)
        owner = torch.arange(self.ne + self.ng, device=xc.device)
        typ[self.gid], owner[self.gid] = self.gtype, self.par
        self.wall, self.recon, self.snb = typ[self.nc] == 5, self.nc < self.ne, owner[self.nc]
        self.dx = self.xc[:, self.nc] - self.xc[:, None, :self.ne]        # (3, face, ne)
        self.active = self.blank == 1
        self.fringe = None if table is None else (_dev(table.fringe, torch.int64) - 1, _dev(table.donor, torch.int64) - 1,
                                                  _dev(table.weight))

    def recover(self, c, pr=None):
        """Primitives of the conserved state and the state they give back."""
        p = self.p
        fsd, k = 4 * p.surfacetension / p.diap, p.pinf * p.gamap
        ug, up = c[1:4] / c[0], c[6:9] / c[5]
        eg, ep = c[4] / c[0] - 0.5 * (ug * ug).sum(0), c[9] / c[5] - 0.5 * (up * up).sum(0)
        g1, g2 = c[0] * (p.gamag - 1) * eg, c[5] * (p.gamap - 1) * ep
        b = (fsd + k) - g1 - g2
        pg = 0.5 * (-b + torch.sqrt(b * b + 4 * (g1 * (fsd + k))))
        pp = pg + fsd
        ag = g1 / pg
        ap = 1 - ag
        tg = pg / (c[0] / ag * R_GAS)
        tp = (pp + p.pinf) * p.gamap / ((p.gamap - 1) * (c[5] / ap) * p.cpp)
        ag, ap, vg, vp = self.blend(ag, ap, torch.cat([ug, tg[None], pg[None]]), torch.cat([up, tp[None], pp[None]]))
        rg, rp = self.densities(vg, vp)
        q = torch.stack([vg[0], vg[1], vg[2], vg[3], vg[4], vp[4], ag, ap, vp[0], vp[1], vp[2], vp[3], rg, rp])
        eg = vg[4] / ((p.gamag - 1) * rg) + 0.5 * (vg[:3] ** 2).sum(0)
        ep = (vp[4] + k) / ((p.gamap - 1) * rp) + 0.5 * (vp[:3] ** 2).sum(0)
        mg, mp = ag * rg, ap * rp
        return q, torch.stack([mg, *(mg * vg[:3]), mg * eg, mp, *(mp * vp[:3]), mp * ep])

    def blend(self, ag, ap, vg, vp):
        lo, hi = self.p.epslnmin, self.p.epslnmax
        m = ag < lo
        ag, ap, vg = torch.where(m, lo, ag), torch.where(m, 1 - lo, ap), torch.where(m, vp, vg)
        m = ap < lo
        ag, ap, vp = torch.where(m, 1 - lo, ag), torch.where(m, lo, ap), torch.where(m, vg, vp)

        def f(a):
            s = (a - lo) / (hi - lo)
            return -(s * s * (2 * s - 3))
        vg = torch.where((ag >= lo) & (ag <= hi), f(ag) * vg + (1 - f(ag)) * vp, vg)
        vp = torch.where((ap >= lo) & (ap <= hi), f(ap) * vp + (1 - f(ap)) * vg, vp)
        return ag, ap, vg, vp

    def densities(self, vg, vp):
        p = self.p
        return vg[4] / (R_GAS * vg[3]), p.gamap * (vp[4] + p.pinf) / ((p.gamap - 1) * p.cpp * vp[3])

    def dtmin(self, q):
        p = self.p
        a = torch.maximum(torch.sqrt(p.gamag * q[PG] / q[RG]), torch.sqrt(p.gamap * (q[PP] + p.pinf) / q[RP]))
        u = torch.maximum((q[UG:WG + 1] ** 2).sum(0).sqrt(), (q[UP:WP + 1] ** 2).sum(0).sqrt())
        return (self.dl / (a + u)).amin()

    def ghosts(self, pr, dt, viscous):
        """Ghost values of the boundary types of these meshes: slip wall 5,
        isothermal wall 6, far field 7, spanwise plane 53."""
        if not self.ng:
            return
        p, t = self.p, self.gtype
        par, old = pr[:, self.par], pr[:, self.gid]
        new = par.clone()
        for k in (UG, VG, WG, UP, VP, WP):
            new[k] = torch.where((t == 5) | (t == 6), -par[k], par[k])
        for k in (TG, TP):
            new[k] = torch.where(t == 6, 2 * p.twall - par[k], par[k])
        far = {UG: p.ugmin, VG: p.vgmin, WG: p.wgmin, UP: p.upmin, VP: p.vpmin, WP: p.wpmin, TG: p.tgmin, TP: p.tpmin,
               PG: p.pmin, PP: p.pmin + 4 * p.surfacetension / p.diap, AP: p.phipzero, AG: 1 - p.phipzero}
        for k, v in far.items():
            new[k] = torch.where(t == 7, torch.full_like(new[k], v), new[k])
        z, out = t == 53, par[WG] > old[WG]
        frac = 1 / (1 + par[WG] * dt / self.dd)
        for k in (UG, VG, TG):
            new[k] = torch.where(z & out, old[k] * frac + (1 - frac) * (2 * par[k] - old[k]), new[k])
        new[WG] = torch.where(z, torch.where(out & viscous, -old[WG], -par[WG]), new[WG])
        new[WP] = torch.where(z, -par[WP], new[WP])
        new[RG], new[RP] = self.densities(new[[UG, VG, WG, TG, PG]], new[[UP, VP, WP, TP, PP]])
        pr[:, self.gid] = new

    def dissipation(self, c, q, dt):
        """JST: pressure, mass and energy switches, second and fourth differences."""
        nb = self.snb
        lap = (c[:, nb] - c[:, None]).sum(1)

        def sw(v, e):
            return (v[nb] - v).abs().sum(0) / ((v[nb] + v).abs().sum(0) + e)
        anu = [sw(q[PG], 0) + sw(c[4], E6) + sw(c[0], E6), sw(q[PP], 0) + sw(c[5], E6) + sw(c[9], E6)]
        w = 0.5 * (self.vol / dt + self.vol[nb] / dt)
        d = torch.empty_like(c)
        for s, a in enumerate(anu):
            e2 = torch.maximum(a, a[nb]) / 16
            e4 = (1 / 1024 - e2).clamp_min(0)
            for k in range(5 * s, 5 * s + 5):
                d[k] = (e2 * w * (c[k][nb] - c[k])).sum(0) - (e4 * w * (lap[k][nb] - lap[k])).sum(0)
        return d

    def viscous(self, pr):
        """Face-centred least squares, Newtonian stresses and heat flux."""
        p, ne = self.p, self.ne
        out = torch.zeros(8, ne, dtype=pr.dtype, device=pr.device)
        own = torch.arange(ne, device=pr.device)
        for f in range(4):
            n = self.nc[f]
            inner = n < ne
            far = self.nc[:, n.clamp_max(ne - 1)]
            pts = torch.cat([self.nc, torch.where(inner, far, own)])                       # (8, ne)
            use = torch.ones_like(pts, dtype=pr.dtype)
            use[5:] = inner.to(pr.dtype)
            x = self.xc[:, pts] - self.fcv[f][:, None]
            A = _normal(x, 1 / use)
            for ph, cols in enumerate(((UG, VG, WG, TG), (UP, VP, WP, TP))):
                mid = [0.5 * (pr[k][:ne] + pr[k][n]) for k in cols]
                g = [_solve(A, ((pr[k][pts] - m) * x * use).sum(1)) for k, m in zip(cols, mid)]
                mu = p.as_ * torch.sqrt(mid[3]) / (1 + p.ts / mid[3]) if ph == 0 else torch.full_like(mid[3], AMU_P)
                cond = mu * p.cpg / p.prg if ph == 0 else mu * p.cpp / PR_P
                div = C23 * (g[0][0] + g[1][1] + g[2][2])
                tau = [[mu * (g[i][j] + g[j][i] - (div if i == j else 0)) for j in range(3)] for i in range(3)]
                heat = [sum(mid[i] * tau[i][j] for i in range(3)) + cond * g[3][j] for j in range(3)]
                a = 0.5 * (pr[AG + ph][:ne] + pr[AG + ph][n])
                for k, v in enumerate((*tau, heat)):
                    out[4 * ph + k] += a * sum(v[j] * self.sc[f][j] for j in range(3))
        return torch.where(self.active, out, 0)

    def gradients(self, pr):
        """1/r^2-weighted least squares of 13 fields, and the limiter."""
        p, ne, x = self.p, self.ne, self.dx
        w = (x * x).sum(0)
        A = _normal(x, w)
        grad = []
        for k in GRAD:
            d = pr[k][self.nc] - pr[k][:ne]
            r = (d * x / w).sum(1)
            if k == TP:                  # the reference leaves the last weight of this sum out
                r[1] += d[3] * x[1, 3] * (1 - 1 / w[3])
            grad.append(_solve(A, r))
        eps = (p.venkat_k * self.dl) ** 3
        rf = self.fch.transpose(0, 1) - self.xc[:, None, :ne]                              # (3, face, ne)
        phi = torch.full_like(self.vol, math.inf)
        for k in (PG, PP, RG, RP):
            v, d = torch.cat([pr[k][None, :ne], pr[k][self.nc]]), (rf * grad[GRAD.index(k)][:, None]).sum(0)
            top, low = v.amax(0) - pr[k][:ne], v.amin(0) - pr[k][:ne]
            m = torch.where(d > 0, top, low)
            one = (((m * m + eps) * d + 2 * d * d * m) / (m * m + 2 * d * d + m * d + eps)) / d
            phi = torch.minimum(phi, torch.where(d == 0, 1.0, one).amin(0))
        ok = self.active
        return torch.where(ok, torch.stack(grad[:11]), 0), torch.where(ok, phi, 0)

    def faces(self, pr, grad, phi):
        """Sum of the face fluxes of every cell, (10, ne)."""
        p, ne = self.p, self.ne
        rhs = torch.zeros(10, ne, dtype=pr.dtype, device=pr.device)
        cols = [UG, VG, WG, TG, PG, UP, VP, WP, TP, PP, AG]
        for f in range(4):
            n = self.nc[f]
            area = (self.sc[f] ** 2).sum(0).sqrt()
            e = self.sc[f] / area
            L, R = pr[cols, :ne], pr[:, n][cols]
            if p.myflux == 3:
                sides = [(*v, q[[RG, RP]]) for v, q in (((L[10], 1 - L[10], L[:5], L[5:10]), pr[:, :ne]),
                                                         ((R[10], 1 - R[10], R[:5], R[5:10]), pr[:, n]))]
            else:
                if p.myorder == 2:
                    j = n.clamp_max(ne - 1)
                    lim = torch.where(self.recon[f], torch.minimum(phi, phi[j]), 0)
                    at = [GRAD.index(k) for k in cols]
                    L = L + lim * (grad[at] * (self.fch[f] - self.xc[:, :ne])).sum(1)
                    R = R + lim * (grad[:, :, j][at] * (self.fch[f] - self.xc[:, n])).sum(1)
                sides = []
                for v in (L, R):
                    ag, ap, vg, vp = self.blend(v[10], 1 - v[10], v[:5], v[5:10])
                    sides.append((ag, ap, vg, vp, torch.stack(self.densities(vg, vp))))
            ph = [self.phase(s, e, k) for k in (0, 1) for s in sides]
            flux = {1: self.zien, 2: self.batten, 3: self.central}[p.myflux](ph, e)
            (ag, ap, vg, vp, _) = sides[0]
            zero = torch.zeros_like(area)
            press = torch.stack([zero, *(ag * vg[4] * e), zero, zero, *(ap * vp[4] * e), zero])
            rhs += torch.where(self.wall[f], press, flux) * area
        return rhs

    def phase(self, side, e, k):
        """(a, rho, p, e, q, c, conserved, flux) of one phase of a face state."""
        p, a, v, rho = self.p, side[k], side[2 + k], side[4][k]
        ke = 0.5 * (v[:3] ** 2).sum(0)
        if k == 0:
            en, c = R_GAS * v[3] / (p.gamag - 1) + ke, torch.sqrt(p.gamag * v[4] / rho)
        else:
            en, c = p.cpp * v[3] / p.gamap + p.pinf / rho + ke, torch.sqrt(p.gamap * (v[4] + p.pinf) / rho)
        q = (v[:3] * e).sum(0)
        cons = a * rho * torch.stack([torch.ones_like(q), *v[:3], en])
        push = a * v[4] * torch.stack([torch.zeros_like(q), *e, q])
        return a, rho, v[4], q, c, cons, cons * q + push, push

    def central(self, ph, e):
        return torch.cat([0.5 * (ph[2 * k][6] + ph[2 * k + 1][6]) for k in (0, 1)])

    def star(self, S, s, contact, pstar, e):
        """Flux of side S through its star state."""
        a, rho, pr, q, c, cons, flux, push = S
        back = a * pstar * torch.stack([torch.zeros_like(q), *e, contact])
        cs = ((q - s) * cons + push - back) / ((contact - s) + E6)
        return flux + s * (cs - cons)

    def pick(self, L, R, sl, sr, contact, pstar, e, left, right):
        F = torch.where(contact > 0, self.star(L, sl, contact, pstar, e), self.star(R, sr, contact, pstar, e))
        return torch.where(left, L[6], torch.where(right, R[6], F))

    def batten(self, ph, e):
        out = []
        for L, R in (ph[:2], ph[2:]):
            sl = torch.minimum(L[3] - L[4], R[3] - R[4]).clamp_max(E8)
            sr = torch.maximum(L[3] + L[4], R[3] + R[4]).clamp_min(E8)
            contact = ((R[2] - L[2] + L[1] * L[3] * (sl - L[3]) - R[1] * R[3] * (sr - R[3])) /
                       (L[1] * (sl - L[3]) - R[1] * (sr - R[3]) + E8))
            pstar = torch.maximum(L[2] + L[1] * (L[3] - sl) * (L[3] - contact), E6 * torch.minimum(L[2], R[2]))
            out.append(self.pick(L, R, sl, sr, contact, pstar, e, sl > 0, sr < 0))
        return torch.cat(out)

    def zien(self, ph, e):
        gl, gr, ll, lr = ph
        sl = torch.stack([s[3] - s[4] for s in ph]).amin(0).clamp_max(E8)
        sr = torch.stack([s[3] + s[4] for s in ph]).amax(0).clamp_min(E8)

        def mix(g, w):
            m = g[0] * g[1] + w[0] * w[1]
            mq = g[0] * g[1] * g[3] + w[0] * w[1] * w[3]
            return m, mq, mq / m, g[0] * g[2] + w[0] * w[2]
        rl, rql, ql, pl = mix(gl, ll)
        rr, rqr, qr, pr = mix(gr, lr)
        contact = (pr - pl + rql * (sl - ql) - rqr * (sr - qr)) / (rl * (sl - ql) - rr * (sr - qr) + E8)
        out = []
        for L, R in ((gl, gr), (ll, lr)):
            pstar = torch.maximum(L[2] + L[1] * (L[3] - sl) * (L[3] - contact), E6 * torch.minimum(L[2], R[2]))
            out.append(self.pick(L, R, sl, sr, contact, pstar, e, sl >= 0, (sr <= 0) & (contact <= 0)))
        return torch.cat(out)

    def sources(self, pr):
        """Drag, heat exchange and interface pressure, (10, ne)."""
        p, ne = self.p, self.ne
        q = pr[:, :ne]
        d = q[UG:WG + 1] - q[UP:WP + 1]
        d2 = (d * d).sum(0)
        ag, ap, rg, rp, dl = q[AG], q[AP], q[RG], q[RP], self.dl
        mu = p.as_ * torch.sqrt(q[TG]) / (1 + p.ts / q[TG])
        drag = 0.44 * ag * (ag - 1) * rg * torch.sqrt(d2) * dl * d
        heat = 6 * ap * mu * p.cpg * 2 * (q[TP] - q[TG]) / (p.prg * dl * dl)
        pint = q[PG] - torch.minimum(2 * (ag * rg * ap * rp) / (ag * rp + ap * rg) * d2, 0.01 * q[PG])
        ui = (ag * rg * q[UG:WG + 1] + (1 - ag) * rp * q[UP:WP + 1]) / (ag * rg + (1 - ag) * rp)
        r = (self.dx ** 2).sum(0).sqrt()
        slope = _solve(_normal(self.dx, r), ((pr[AG][self.nc] - ag) * self.dx / r).sum(1))
        mom = drag + pint * slope
        en = pint * (ui * slope).sum(0) + (ui * drag).sum(0) + heat
        zero = torch.zeros_like(en)
        return torch.stack([zero, *-mom, -en, zero, *mom, en]) * self.vol

    def run(self, cu, gp, steps):
        p, ne = self.p, self.ne
        c = _dev(cu)
        pr = torch.zeros(14, ne + self.ng, dtype=c.dtype, device=c.device)
        if self.ng:
            for k, v in zip((UG, VG, WG, PG, TG, RG), _dev(gp)):
                pr[k, self.gid] = v
        time, told = 0.0, []
        pr[:, :ne], c = self.recover(c)
        old = c
        for _ in range(steps):
            start = old                                          # the state that the last step ended with
            if told:
                pr[:, :ne], c = self.recover(start)
            else:
                start = _dev(cu)
            dt = p.cfl * torch.clamp_max(self.dtmin(pr[:, :ne]), 1e8)
            time = time + dt
            extra = self.dissipation(c, pr[:, :ne], dt)
            self.ghosts(pr, dt, True)
            if not p.inviscid:
                v = self.viscous(pr)
                extra[1:5] += v[:4]
                extra[6:10] += v[4:]
            first = None
            for stage in range(4 if p.rk_scheme == 0 else 3):
                pr[:, :ne], c = self.recover(c)
                self.ghosts(pr, dt, False)
                grad, phi = self.gradients(pr) if p.myorder == 2 and p.myflux != 3 else (None, None)
                res = dt / self.vol * (self.faces(pr, grad, phi) + self.sources(pr) - extra)
                if p.rk_scheme == 0:
                    new = (c if stage else start) - 11 / 20 * res
                    first = new if stage == 0 else first
                    new = [new, 3 / 8 * start + 5 / 8 * new, 4 / 9 * start + 5 / 9 * new,
                           111 / 1331 * start + 260 / 1331 * first + 960 / 1331 * new][stage]
                else:
                    new = (c if stage else start) - res
                    new = [new, 0.75 * start + 0.25 * new, start / 3 + 2 / 3 * new][stage]
                c = torch.where(self.active, new, c)
                if self.fringe is not None:
                    i, donor, w = self.fringe
                    c[:, i] = (c[:, donor] * w).sum(2)
            q, c = self.recover(c)
            told.append((time, dt, (q[UG:WG + 1, 0] ** 2).sum().sqrt(), (c[:4] - start[:4]).abs().amax(1)))
            old = c
        ghost = pr[[UG, VG, WG, PG, TG, RG]][:, self.gid]
        cols = [torch.stack([torch.as_tensor(t[k], device=c.device) for t in told]).cpu() for k in range(4)]
        return {"cu": old.cpu(), "ghosts": ghost.cpu(), "time": cols[0], "dt": cols[1], "velmag": cols[2], "diff": cols[3],
                "nan_cells": torch.zeros(steps, dtype=torch.float64)}
