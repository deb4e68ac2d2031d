"""Device memory of a handle: no more bytes per cell than a handle took when
its geometry tables were those of the cells alone (the limits below, measured
on two meshes with hp_estimate_bytes), so every mesh and batch that fitted
then fits; and what a handle takes is what the estimate says."""
import ctypes

import pytest

from hydraphase import PREC_FP64, PREC_FP64_PARITY, PREC_MIXED, Case, cases, lib
from hydraphase._lib import HpMesh
from hydraphase.engine import MeshArrays, estimate_batch_bytes, estimate_bytes

PREC_FP32 = 3


def _spec(name):
    if name == "box":          # inviscid, 24,576 cells, 3,072 ghosts
        return cases.shock_bubble(n=16, alpha_min=0.1)
    if name == "cylinder":     # viscous, 36,864 cells, 7,168 ghosts
        return cases.cylinder(nr=24, nt=64, nz=4)
    return cases.with_dispersed(cases.shock_bubble(n=12, alpha_min=0.1), rad=(2e-4, 3e-4, 4e-4))


# bytes per cell, rounded down
LIMITS = [
    ("box", PREC_FP64_PARITY, {}, 1840), ("box", PREC_FP64, {}, 1840), ("box", PREC_MIXED, {}, 1888),
    ("box", PREC_FP32, {}, 1888), ("box", PREC_MIXED, dict(face_mode=1), 1755),
    ("box", PREC_MIXED, dict(face_mode=2), 1987),
    ("cylinder", PREC_FP64_PARITY, {}, 1953), ("cylinder", PREC_FP64, {}, 1953), ("cylinder", PREC_MIXED, {}, 1999),
    ("cylinder", PREC_MIXED, dict(face_mode=1), 1863), ("cylinder", PREC_MIXED, dict(face_mode=3), 2103),
    ("cylinder", PREC_FP64_PARITY, dict(myflux=3), 1953), ("cylinder", PREC_MIXED, dict(myflux=3), 1999),
    ("box", PREC_MIXED, dict(wall_fp64_layers=4), 2194), ("box", PREC_FP32, dict(wall_fp64_layers=4), 2194),
    ("box", PREC_MIXED, dict(wall_fp64_layers=4, face_mode=1), 2061),
    ("box", PREC_MIXED, dict(wall_fp64_layers=100), 2194),
    ("cylinder", PREC_MIXED, dict(wall_fp64_layers=4), 2324), ("cylinder", PREC_MIXED, dict(wall_fp64_layers=100), 2324),
    ("cylinder", PREC_MIXED, dict(wall_fp64_layers=4, face_mode=1), 2187),
    ("cylinder", PREC_MIXED, dict(wall_fp64_layers=4, myflux=3), 2324),
    ("cylinder", PREC_MIXED, dict(wall_fp64_layers=4, face_mode=2), 2429),
    ("dispersed", PREC_MIXED, dict(wall_fp64_layers=4), 3073),
    ("dispersed", PREC_FP64_PARITY, {}, 2709), ("dispersed", PREC_MIXED, {}, 2756),
]


@pytest.mark.parametrize("name,precision,over,limit", LIMITS)
def test_bytes_per_cell(name, precision, over, limit):
    sp = _spec(name)
    p = sp.params(precision=precision, **over)
    assert estimate_bytes(sp.mesh, p) // sp.mesh.neles <= limit
    assert estimate_batch_bytes([sp.mesh] * 3, p) // (3 * sp.mesh.neles) <= limit


def _aliased(mesh):
    el, gh = mesh.elem.copy(), mesh.ghost.copy()
    new = gh[:, 1] - 3
    for g in range(gh.shape[0]):
        el[gh[g, 0] - 1, 4 + gh[g, 3] - 1] = new[g]
    gh[:, 1] = new
    return MeshArrays(mesh.x, mesh.y, mesh.z, el, gh)


def test_sizes_alone_give_an_upper_bound():
    for name in ("box", "cylinder", "dispersed"):
        sp = _spec(name)
        for precision in (PREC_FP64_PARITY, PREC_MIXED):
            for layers in (0, 4, 100):
                p = sp.params(precision=precision, wall_fp64_layers=layers)
                hm, b = HpMesh(sp.mesh.nodes, sp.mesh.neles, sp.mesh.nghosts, 0, None, None, None, None, None), \
                    ctypes.c_int64()
                assert lib().hp_estimate_bytes(ctypes.byref(hm), ctypes.byref(p), ctypes.byref(b)) == 0
                assert b.value >= estimate_bytes(sp.mesh, p)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [PREC_FP64_PARITY, PREC_MIXED])
@pytest.mark.parametrize("over", [{}, dict(inviscid=1), dict(myflux=3), dict(face_mode=1), dict(wall_fp64_layers=2),
                                  dict(wall_fp64_layers=99), dict(wall_fp64_layers=2, face_mode=1), "aliased"])
def test_a_handle_takes_what_the_estimate_says(precision, over):
    sp = cases.cylinder(nr=4, nt=16, nz=2)
    mesh = _aliased(sp.mesh) if over == "aliased" else sp.mesh
    p = sp.params(precision=precision, **({} if over == "aliased" else over))
    with Case(mesh, p) as c:
        assert c.info()["device_bytes"] <= estimate_bytes(mesh, p)
