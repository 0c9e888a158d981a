"""A wait of a sync-free LU-SGS sweep that runs out inside a solve: a row left
out of the forward order never writes its result, the rows that need it give up
after a short bound, the solve says so, and the next one is as before."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases

from test_gpu_parity import perturb  # noqa: E402

pytestmark = pytest.mark.gpu

LUSGS = 1  # ICS_PC_LUSGS

CALLS = {
    "solve": lambda h, b: h.solve_increment()[1],
    "precondition": lambda h, b: h.precondition(b),
    "tangent": lambda h, b: h.tangent_solve(b, preconditioner=LUSGS, pseudo_time=1, max_cycles=2)[0],
    "adjoint": lambda h, b: h.adjoint_solve(b, preconditioner=LUSGS, pseudo_time=1, max_cycles=2)[0],
}


# blocks in FP64 and FP32 (16 and 4 lanes a row, and FP32 blocks on FP64 vectors)
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("call", list(CALLS))
def test_solves_report_the_timeout(gpu_binding, call, precision):
    w = perturb(cases.bump_channel(12, 6, 4, ordering_mode="natural"))
    h = abi.CaseHandle(gpu_binding, w.mesh, cases.make_config(gpu_binding, w.settings, precision=precision, max_iter=2))
    h.set_primitive(w.p, w.U, w.T)
    b = h.residual()
    h.assemble_jacobian()
    before = CALLS[call](h, b)
    h.test_sweep_wait(0, 1000)  # cell 0 has upper neighbours
    with pytest.raises(abi.IcsError) as e:
        CALLS[call](h, b)
    assert e.value.status == abi.ICS_ERR_TIMEOUT
    h.test_sweep_wait(0, 0)
    assert np.array_equal(before, CALLS[call](h, b))
