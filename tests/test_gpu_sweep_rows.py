"""LU-SGS sweeps of rows with more than three neighbours on a side (a random
numbering) and with the viscous part of the blocks, in both precisions and with
FP32 blocks, against the sequential oracle."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _open(binding, w, **over):
    h = abi.CaseHandle(binding, w.mesh, cases.make_config(binding, w.settings, **over))
    h.set_primitive(w.p, w.U, w.T)
    h.residual()
    h.assemble_jacobian()
    return h


# a row is a few dozen products and its round-off grows by at most the number
# of levels (< 30): 30 * 100 * 2^-53 < 1e-12; FP32 blocks and results 1e-5, as
# for the other schedules
@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (1, 1e-5)])
@pytest.mark.parametrize("n,over", [(3, {}), (7, {}), (13, {}), (7, {"viscous_lf_jacobian": 0})])
def test_random_numbering(oracle_binding, gpu_binding, n, over, precision, tol):
    w = cases.random_box(n, ordering_mode="natural")
    assert np.bincount(w.mesh.neighbour, minlength=w.mesh.n_cells).max() > 3 or n < 7
    hg, ho = _open(gpu_binding, w, precision=precision, **over), _open(oracle_binding, w, **over)
    r = np.random.default_rng(5).standard_normal((w.mesh.n_cells, 5))
    a, b = hg.precondition(r), ho.precondition(r)
    assert np.abs(a - b).max() <= tol * np.abs(b).max()
