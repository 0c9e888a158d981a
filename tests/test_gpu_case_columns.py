"""Gram-Schmidt columns of stacked cases at the sizes where their clusters'
registers run out: one and many entries per thread, the largest case of each
instance and one cell more, small and large cases in one stack."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _tube(n):
    w = cases.shock_tube(n, ordering_mode="colour")
    rng = np.random.default_rng(n)
    w.p = w.p * (1 + 0.02 * rng.uniform(-1, 1, n))
    w.T = w.T * (1 + 0.02 * rng.uniform(-1, 1, n))
    w.U[:, 0] += 30.0 * rng.uniform(-1, 1, n)
    return w


def _increment(binding, w, precision, delta_t, start=None):
    h = abi.CaseHandle(binding, w.mesh, cases.make_config(binding, w.settings, precision=precision, max_iter=1,
                                                          delta_t=delta_t))
    if start is not None:
        h.set_cases(start)
    h.set_primitive(w.p, w.U, w.T)
    h.begin_time_step()
    h.residual()
    h.assemble_jacobian()
    _, dW, _ = h.solve_increment()
    return dW


# One restart cycle of each case in the stack against a handle of its own,
# whose columns add up in another order: FP64 1e-10 of the largest entry of
# each equation, mixed 1e-3 (2^-24 per operation over eight directions), as the
# columns of one system are held to
@pytest.mark.parametrize("precision,tol", [(0, 1e-10), (1, 1e-3)])
@pytest.mark.parametrize("sizes", [(3, 64, 1638), (5, 1639, 6553), (410, 6554, 13107), (13107, 51, 13108)])
def test_columns_follow_a_handle_of_their_own(gpu_binding, sizes, precision, tol):
    ws = [_tube(n) for n in sizes]
    dt = 1e-2 / max(sizes)
    w, start = cases.stack_cases(ws)
    dW = _increment(gpu_binding, w, precision, dt, start)
    for k, own in enumerate(ws):
        a, b = dW[start[k]:start[k + 1]], _increment(gpu_binding, own, precision, dt)
        scale = np.abs(b).max(axis=0)
        assert (np.abs(a - b) <= tol * np.maximum(scale, 1e-300)).all(), sizes[k]
