"""FP64 products and sweeps of few rows on five lanes per row, and the
row-per-thread kernels beyond: fewer rows than a warp takes, a warp's six and
one more, a block's twelve and one more, and both sides of the limit of 36000
rows (of the product, 36000 cells; of a level of two colours, 72000)."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _open(binding, w, **over):
    h = abi.CaseHandle(binding, w.mesh, cases.make_config(binding, w.settings, precision=0, max_iter=1, **over))
    rng = np.random.default_rng(w.mesh.n_cells)
    n = w.mesh.n_cells
    h.set_primitive(w.p * (1 + 0.02 * rng.uniform(-1, 1, n)), w.U, w.T * (1 + 0.02 * rng.uniform(-1, 1, n)))
    h.residual()
    h.assemble_jacobian()
    return h


# a row is at most 7 x 5 products: 35 * 2^-53 of their largest, with a factor
# 100 for the blocks' spread over the equations, < 1e-12; the increments of one
# restart cycle 1e-10, as in the other parity tests
@pytest.mark.parametrize("shape", [(2, 1, 1), (3, 2, 1), (4, 3, 1), (5, 5, 1), (13, 1, 1), (9, 5, 3),
                                   (100, 36, 10), (77, 39, 12), (100, 36, 20), (2001, 36, 1)])
def test_rows_follow_the_oracle(oracle_binding, gpu_binding, shape):
    w = cases.bump_channel(*shape, ordering_mode="colour", second_order=False)
    hg, ho = _open(gpu_binding, w), _open(oracle_binding, w)
    x = np.random.default_rng(3).standard_normal((w.mesh.n_cells, 5))
    for f in ("matrix_mul", "precondition"):
        a, b = getattr(hg, f)(x), getattr(ho, f)(x)
        assert (np.abs(a - b) <= 1e-12 * np.abs(b).max(axis=0)).all(), f
    dg, do = hg.solve_increment()[1], ho.solve_increment()[1]
    scale = np.abs(do).max(axis=0)
    scale[1:4] = scale[1:4].max()  # the momentum components share one scale
    assert (np.abs(dg - do) <= 1e-10 * scale).all()


def test_viscous_blocks_of_few_rows(oracle_binding, gpu_binding):
    w = cases.random_box(6, ordering_mode="rcm+colour")
    hg, ho = _open(gpu_binding, w, viscous_lf_jacobian=0), _open(oracle_binding, w, viscous_lf_jacobian=0)
    x = np.random.default_rng(3).standard_normal((w.mesh.n_cells, 5))
    for f in ("matrix_mul", "precondition"):
        a, b = getattr(hg, f)(x), getattr(ho, f)(x)
        assert (np.abs(a - b) <= 1e-12 * np.abs(b).max(axis=0)).all(), f
