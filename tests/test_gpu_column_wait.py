"""A wait of a Gram-Schmidt column that runs out: a block left out of the
exchange never publishes its sum, the others give up after a short bound, every
solve that uses the columns says so, and the next one is as before."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases

from test_gpu_parity import perturb  # noqa: E402

pytestmark = pytest.mark.gpu


def _solve(h, allow=(abi.ICS_OK,)):
    h.residual()
    h.assemble_jacobian()
    return h.solve_increment(allow)


# a column of one block (no wait), of two and of a block per SM
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape,waits", [((5, 3, 3), False), ((16, 8, 4), True), ((61, 31, 29), True)])
def test_solve_reports_the_timeout(gpu_binding, shape, waits, precision):
    w = perturb(cases.bump_channel(*shape, ordering_mode="colour"))
    h = abi.CaseHandle(gpu_binding, w.mesh, cases.make_config(gpu_binding, w.settings, precision=precision, max_iter=3))
    h.set_primitive(w.p, w.U, w.T)
    _, before, _ = _solve(h)
    h.test_column_wait(1000)
    _, _, status = _solve(h, (abi.ICS_OK, abi.ICS_ERR_TIMEOUT))
    assert status == (abi.ICS_ERR_TIMEOUT if waits else abi.ICS_OK)
    h.test_column_wait(0)
    _, after, _ = _solve(h)
    assert np.array_equal(before, after)


def test_scalar_transport_reports_the_timeout(gpu_binding):
    w = cases.bump_channel(16, 8, 4, ordering_mode="colour")
    h = abi.CaseHandle(gpu_binding, w.mesh, cases.make_config(gpu_binding, w.settings))
    h.set_primitive(w.p, w.U, w.T)
    fixed = np.array([p.kind in (3, 5) for p in w.mesh.patches], np.int32)
    h.scalar_enable(0.5 + 0.4 * np.sin(3.0 * w.mesh.C[:, 0]), fixed, np.where(fixed, 0.9, 0.0), D=2e-5, recon=3)
    h.residual()
    h.test_column_wait(1000)
    before = h.get_scalar()[0]
    with pytest.raises(abi.IcsError) as e:
        h.scalar_transport(1)
    assert e.value.status == abi.ICS_ERR_TIMEOUT
    assert np.array_equal(before, h.get_scalar()[0])  # no partial increment
    h.test_column_wait(0)
    h.scalar_transport(1)
    assert np.isfinite(h.get_scalar()[0]).all()
