"""Which handles recover the next stage's primitives in the flux kernel: the
mixed variant's plain handle launches the primitive pass once per step, one with
a halo table in every stage, hp_info counts those launches, and the two routes
leave the same bits in the face modes that add in a fixed order."""
import ctypes

import numpy as np
import pytest

from hydraphase import PREC_MIXED, Batch, Case, cases
from hydraphase._lib import KERNEL_KINDS

pytestmark = pytest.mark.gpu


def _counts(L, h, steps):
    """(launches of the primitive pass per step, kernels per step)"""
    n = len(KERNEL_KINDS)
    ms, cnt = (ctypes.c_double * n)(), (ctypes.c_int64 * n)()
    assert L.hp_profile_steps(h, steps, ms, cnt, n) == 0
    k = ctypes.c_int64()
    assert L.hp_info(h, ctypes.byref(k), None, None) == 0
    return cnt[KERNEL_KINDS.index("prim_stage")] / steps, k.value


@pytest.mark.parametrize("rk,nstage", [(0, 4), (1, 3)])
@pytest.mark.parametrize("face_mode", [0, 2])
def test_routes_and_their_launches(rk, nstage, face_mode):
    sp = cases.shock_bubble_on(cases.box_mesh(5, 7, 11, jitter=0.1, seed=2, bc_type=5), alpha_min=0.1)
    over = dict(precision=PREC_MIXED, rk_scheme=rk, face_mode=face_mode, cfl=0.05)
    with Case(sp.mesh, sp.params(**over)) as c:
        c.set_state(0.0, sp.cu, sp.ghost_prims)
        c.step(3)
        plain = c.state()[1]
        prim, kernels = _counts(c.L, c.h, 2)
        assert prim == 1
    # case 1, its cell 1 frozen, takes case 0's cell 1: nothing of consequence
    frozen = cases.MeshArrays(sp.mesh.x, sp.mesh.y, sp.mesh.z, sp.mesh.elem.copy(), sp.mesh.ghost)
    frozen.elem[0, 8] = 3
    with Batch([sp.mesh, frozen], sp.params(**over)) as b:
        one, zero = np.ones(1, np.int32), np.zeros(1, np.int32)
        ip = ctypes.POINTER(ctypes.c_int32)
        assert b.L.hp_set_halo(b.h, 1, one.ctypes.data_as(ip), one.ctypes.data_as(ip), zero.ctypes.data_as(ip),
                               one.ctypes.data_as(ip)) == 0
        for k in (0, 1):
            b.set_state(k, 0.0, sp.cu, sp.ghost_prims)
        b.step(3)
        apart = b.state(0)[1]
        prim, kernels_apart = _counts(b.L, b.h, 2)
        assert prim == nstage
    assert kernels_apart - kernels == (nstage - 1) + nstage     # primitive passes, and the halo copy of each stage
    np.testing.assert_array_equal(apart, plain)
