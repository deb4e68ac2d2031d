"""The fused step runs with three blocks per SM on small meshes and with four
on others: both give the separate launches' state bit for bit, on both sides of
the line and with both HLLC solvers."""
import numpy as np
import pytest

from hydraphase import PREC_FP64_PARITY, Case, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("myflux", [1, 2])
@pytest.mark.parametrize("n", [1, 21, 22])     # 6, 55,566 and 63,888 cells; the line is at 56,832
def test_fused_step_equals_separate_launches(n, myflux):
    spec = cases.shock_bubble(n=n, alpha_min=0.1)
    out = []
    for use_graph in (1, 2):
        with Case(spec.mesh, spec.params(precision=PREC_FP64_PARITY, use_graph=use_graph, myflux=myflux, cfl=0.1)) as c:
            c.set_state(0.0, spec.cu, spec.ghost_prims)
            dt = c.step(3)["dt"]
            out.append((c.state()[1], dt, c.info()["kernels_per_step"]))
    np.testing.assert_array_equal(out[1][0], out[0][0])
    np.testing.assert_array_equal(out[1][1], out[0][1])
    assert out[1][2] == 1
