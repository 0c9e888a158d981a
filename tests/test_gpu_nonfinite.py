"""The residual's finite check where a single cell or a single equation is not
finite: the first and the last cell of a mesh whose size fills no block, and an
energy flux that overflows while the mass flux and its squares do not."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _run(binding, cell, entry, value, precision=0):
    w = cases.bump_channel(9, 5, 3, ordering_mode="colour")
    h = abi.CaseHandle(binding, w.mesh, cases.make_config(binding, w.settings, precision=precision))
    h.set_primitive(w.p, w.U, w.T)
    clean = h.residual()
    W = h.get_state()["W"]
    W[cell, entry] = value
    h.set_conservative(W)
    with pytest.raises(abi.IcsError) as e:
        h.residual()
    assert e.value.status == abi.ICS_ERR_NONFINITE
    # the flag of one evaluation does not reach the next
    h.set_primitive(w.p, w.U, w.T)
    assert np.isfinite(h.residual()).all()
    return clean


@pytest.mark.parametrize("cell", [0, -1])
@pytest.mark.parametrize("entry,value", [(4, np.nan), (4, np.inf), (4, 1e308), (1, 1e110)])
def test_one_cell_is_found(gpu_binding, oracle_binding, cell, entry, value):
    _run(oracle_binding, cell, entry, value)
    _run(gpu_binding, cell, entry, value)
