"""Scalar transport on a few cells of a handle in mixed precision: its FP64
Krylov basis is larger there than the FP32 basis of the flow's solve."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _scalar(b, n, precision, directions):
    w = cases.shock_tube(n)
    h = abi.CaseHandle(b, w.mesh, cases.make_config(b, w.settings, precision=precision,
                                                          n_directions=directions))
    h.set_primitive(w.p, w.U + 10.0, w.T)
    P = len(w.mesh.patches)
    h.scalar_enable(0.3 + 0.1 * np.sin(np.arange(n)), np.zeros(P, np.int32), np.zeros(P))
    h.begin_time_step()
    h.residual()
    h.scalar_transport(1)
    return h.get_scalar()[0]


# the scalar's matrix, right-hand side and solve are FP64 in both precisions and
# start from the same FP64 flow: the same bits.  (Fewer directions than cells:
# a space that closes earlier is an error.)
@pytest.mark.parametrize("n,directions", [(2, 1), (3, 2), (7, 6), (12, 8), (13, 8), (25, 8)])
def test_few_cells_in_mixed_precision(gpu_binding, oracle_binding, n, directions):
    mixed = _scalar(gpu_binding, n, 1, directions)
    assert np.array_equal(mixed, _scalar(gpu_binding, n, 0, directions))
    assert np.abs(mixed - _scalar(oracle_binding, n, 0, directions)).max() < 1e-9
