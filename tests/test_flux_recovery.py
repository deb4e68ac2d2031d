"""The mixed variant's flux kernel recovers the next stage's primitives itself
where nothing else changes the state between the stages; handles with a
partition halo, an overset fringe or an exchange callback keep the separate
pass.  Both routes are the same formulas: a handle with a halo table that
copies nothing of consequence (one cell of a second, identical case onto its
frozen twin) must march like the plain one.  Sizes: one block, remainders of
the 128-thread blocks, and several blocks; both RK schemes and the face modes
with a face list."""
import ctypes

import numpy as np
import pytest

from hydraphase import PREC_MIXED, Batch, Case, cases

pytestmark = pytest.mark.gpu


def _spec(n):
    sp = cases.shock_bubble_on(cases.box_mesh(*n, jitter=0.1, seed=2, bc_type=5), alpha_min=0.1)
    sp.flow["cfl"] = 0.05
    return sp


def _close(a, b, tol):
    rho_a, rho_b = a[0] + a[5], b[0] + b[5]
    assert np.linalg.norm(rho_a - rho_b) <= tol * np.linalg.norm(rho_b)
    for k in (4, 9):
        assert np.linalg.norm(a[k] - b[k]) <= tol * np.linalg.norm(b[k])


@pytest.mark.parametrize("n", [(1, 3, 7), (3, 4, 5), (5, 7, 11)])
@pytest.mark.parametrize("rk", [0, 1])
@pytest.mark.parametrize("face_mode", [0, 2, 3])
def test_recovery_in_the_flux_kernel(n, rk, face_mode):
    sp = _spec(n)
    over = dict(rk_scheme=rk, face_mode=face_mode)
    with Case(sp.mesh, sp.params(precision=PREC_MIXED, **over)) as c:
        c.set_state(0.0, sp.cu, sp.ghost_prims)
        fused = c.info()["kernels_per_step"]
        d = c.step(3)
        _, cu, _ = c.state()
    # two cases coupled by a halo: the second case's cell 1, frozen, takes the
    # first case's cell 1
    frozen = cases.MeshArrays(sp.mesh.x, sp.mesh.y, sp.mesh.z, sp.mesh.elem.copy(), sp.mesh.ghost)
    frozen.elem[0, 8] = 3
    with Batch([sp.mesh, frozen], sp.params(precision=PREC_MIXED, **over)) as b:
        one = np.ones(1, np.int32)
        zero = np.zeros(1, np.int32)
        ip = ctypes.POINTER(ctypes.c_int32)
        assert b.L.hp_set_halo(b.h, 1, one.ctypes.data_as(ip), one.ctypes.data_as(ip), zero.ctypes.data_as(ip),
                               one.ctypes.data_as(ip)) == 0
        for k in (0, 1):
            b.set_state(k, 0.0, sp.cu, sp.ghost_prims)
        b.step(3)
        _, apart, _ = b.state(0)
    assert np.isfinite(cu).all() and (d["nan_cells"] == 0).all() and fused > 0
    # FP64 recovery of the same state: roundings of FP64 only (face mode 3 adds
    # in any order)
    _close(cu, apart, 1e-9 if face_mode != 3 else 1e-6)
