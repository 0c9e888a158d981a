"""A Krylov space that closes before the cycle's last direction: the vector left
over is exactly zero, its division by its norm is not finite, and the solve says
so -- on a fresh handle as after other solves, whatever the basis held."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solves_before", [0, 3])
def test_a_closed_space_is_reported(gpu_binding, solves_before):
    n = 1  # the scalar's system of one cell closes after one direction
    w = cases.shock_tube(n)
    h = abi.CaseHandle(gpu_binding, w.mesh, cases.make_config(gpu_binding, w.settings, n_directions=4))
    h.set_primitive(w.p, w.U + 10.0, w.T)
    P = len(w.mesh.patches)
    h.scalar_enable(np.full(n, 0.3), np.zeros(P, np.int32), np.zeros(P))
    h.begin_time_step()
    h.residual()
    for _ in range(solves_before):
        h.assemble_jacobian()
        h.solve_increment(allow=(abi.ICS_OK, abi.ICS_ERR_NONFINITE, abi.ICS_ERR_BREAKDOWN))
    with pytest.raises(abi.IcsError) as e:
        h.scalar_transport(1)
    assert e.value.status == abi.ICS_ERR_NONFINITE
