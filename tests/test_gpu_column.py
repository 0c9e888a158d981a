"""Gram-Schmidt columns of the GMRES cycle at the sizes where their grid,
chunks and registers run out: less than a 16-byte chunk per thread, a partial
last chunk, one and many blocks, slices longer than the registers hold."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _increment(binding, n, precision):
    w = cases.shock_tube(n, ordering_mode="colour")
    rng = np.random.default_rng(n)
    w.p = w.p * (1 + 0.02 * rng.uniform(-1, 1, n))
    w.T = w.T * (1 + 0.02 * rng.uniform(-1, 1, n))
    w.U[:, 0] += 30.0 * rng.uniform(-1, 1, n)
    h = abi.CaseHandle(binding, w.mesh, cases.make_config(binding, w.settings, precision=precision, max_iter=1,
                                                          delta_t=1e-2 / n))
    h.set_primitive(w.p, w.U, w.T)
    h.begin_time_step()
    h.residual()
    h.assemble_jacobian()
    _, dW, _ = h.solve_increment()
    return dW


# FP64 sums in another order: the tolerance of increments against the oracle
# (1e-10 of the largest entry of each equation)
@pytest.mark.parametrize("n", [3, 7, 51, 64, 1023, 13107, 26215])
def test_increments_follow_the_oracle(oracle_binding, gpu_binding, n):
    a, b = _increment(gpu_binding, n, 0), _increment(oracle_binding, n, 0)
    scale = np.abs(b).max(axis=0)
    assert (np.abs(a - b) <= 1e-10 * np.maximum(scale, 1e-300)).all()


# FP32 against FP64 on the device: one restart cycle of eight directions with
# 2^-24 per operation, 1e-3 of the largest entry (increments of the mixed path
# are held to 5e-3); 1,200,001 cells leave part of every slice outside the
# registers in both precisions
@pytest.mark.parametrize("n", [5, 53, 4099, 120001, 500009, 1200001])
def test_mixed_increments_follow_fp64(gpu_binding, n):
    a, b = _increment(gpu_binding, n, 1), _increment(gpu_binding, n, 0)
    scale = np.abs(b).max(axis=0)
    assert (np.abs(a - b) <= 1e-3 * np.maximum(scale, 1e-300)).all()
