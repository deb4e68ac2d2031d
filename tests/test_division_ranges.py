"""Meshes whose geometry leaves the range in which the FP64 kernels' shared-
reciprocal division is exact: the set-up bits (least-squares weights and
determinants, centroid differences, face areas) and the viscous kernel's own
test then send cells to hardware division, and the parity variant still equals
the CPU oracle bit for bit.  Box meshes scaled by powers of two (all axes, or z
alone), each in one handle with the unscaled mesh, so that warps hold cells in
and out of range."""
import numpy as np
import pytest

import oracle as O
from hydraphase import PREC_FP64_PARITY, Batch, cases
from hydraphase.engine import MeshArrays

pytestmark = pytest.mark.gpu

STEPS = 2


def _scaled(b, s):
    m = b.mesh
    return MeshArrays(m.x * s[0], m.y * s[1], m.z * s[2], m.elem, m.ghost)


# scales of x, y, z and whether viscous terms run (on the smallest meshes they
# would outgrow the acoustic time step): the viscous normal matrix's determinant
# 2^-110; weights 2^-124; weights, differences and areas far below; one thin axis
# with determinants 2^-300 and 2^-1000
SCALES = {"viscous": ((2.0 ** -18,) * 3, True), "weights": ((2.0 ** -60,) * 3, False),
          "small": ((2.0 ** -120,) * 3, False), "thin": ((1.0, 1.0, 2.0 ** -150), False),
          "very thin": ((1.0, 1.0, 2.0 ** -500), False)}


@pytest.mark.parametrize("myflux", [1, 2])
@pytest.mark.parametrize("name", list(SCALES))
def test_parity_out_of_range(name, myflux):
    built = cases.box_mesh(4, 4, 3, jitter=0.1, seed=4, bc_type=5)
    spec = cases.shock_bubble_on(built, alpha_min=0.1, reference_scheme=True)
    scale, viscous = SCALES[name]
    meshes = [_scaled(built, scale), built.mesh]
    # (as_ = 0: no interphase heat, which goes with 1 / dl^2)
    over = dict(myflux=myflux, cfl=0.05, inviscid=0 if viscous else 1, as_=0.0)
    ref = []
    for m in meshes:
        orc = O.Oracle(O.params_from_flow(spec.flow, **{**spec.extra, **over}), O.Mesh(m.x, m.y, m.z, m.elem, m.ghost))
        orc.set_state(0.0, spec.cu, spec.ghost_prims)
        t = orc.run(STEPS)[0]
        ref.append((t, orc.cu()[:, :m.neles], orc.ghost_restart()))
        assert np.isfinite(ref[-1][1]).all() and np.isfinite(t).all() and (ref[-1][1] != spec.cu).mean() > 0.5
    with Batch(meshes, spec.params(precision=PREC_FP64_PARITY, **over)) as b:
        for k in (0, 1):
            b.set_state(k, 0.0, spec.cu, spec.ghost_prims)
        b.step(STEPS)
        for k in (0, 1):
            _, got, gp = b.state(k)
            np.testing.assert_array_equal(got, ref[k][1])
            np.testing.assert_array_equal(gp, ref[k][2])
