"""Norm factors and residuals of the linear solver at the sizes where the
reductions' grid changes: part of a block, one block, a block and one cell,
every block full, and one cell more than that."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _solve(binding, n, precision):
    w = cases.shock_tube(n, ordering_mode="colour")
    rng = np.random.default_rng(n)
    w.p = w.p * (1 + 0.02 * rng.uniform(-1, 1, n))
    w.T = w.T * (1 + 0.02 * rng.uniform(-1, 1, n))
    w.U[:, 0] += 30.0 * rng.uniform(-1, 1, n)
    h = abi.CaseHandle(binding, w.mesh, cases.make_config(binding, w.settings, precision=precision, max_iter=1,
                                                          delta_t=1e-2 / n))
    h.set_primitive(w.p, w.U, w.T)
    h.begin_time_step()
    b = h.residual()
    h.assemble_jacobian()
    perf, dW, _ = h.solve_increment()
    W = h.get_state()["W"]
    t = h.matrix_mul(W - W.mean(axis=0))
    nf = [np.abs(t[:, 0]).sum() + np.abs(b[:, 0]).sum(),
          np.linalg.norm(t[:, 1:4], axis=1).sum() + np.linalg.norm(b[:, 1:4], axis=1).sum(),
          np.abs(t[:, 4]).sum() + np.abs(b[:, 4]).sum()]
    nf = np.array([nf[0], nf[1], nf[1], nf[1], nf[2]])
    r = b - h.matrix_mul(dW)
    return (np.array(perf.init_res[:5]), np.abs(b).sum(axis=0) / nf, np.array(perf.final_res[:5]),
            np.abs(r).sum(axis=0) / nf)


# Against numpy's sums of the same terms.  FP64: the sums differ by a few
# rounding errors, the average of W by one that (W - avg W), 1e-2 of W, sees a
# hundredfold: 1e-12.  Mixed: A (W - avg W) in FP32, 1e-4 of the initial
# residuals (2^-24 over the 15 products of a row and their cancellation).  The
# final ones are differences b - A x, whose 15 products of a row (up to 100
# times b in the density and energy rows) each round by 2^-53 or 2^-24
@pytest.mark.parametrize("n", [2, 255, 256, 257, 155648, 155649])
@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (1, 1e-4)])
def test_residual_norms(gpu_binding, n, precision, tol):
    init, ref_init, final, ref_final = _solve(gpu_binding, n, precision)
    assert (np.abs(init - ref_init) <= tol * np.maximum(ref_init, 1e-300)).all(), (init, ref_init)
    noise = 15 * 100 * 2.0 ** (-53 if precision == 0 else -24) * ref_init.max()
    assert (np.abs(final - ref_final) <= tol * ref_final + noise).all(), (final, ref_final)
