"""LU-SGS sweeps of every schedule against the sequential oracle, at the sizes
where the schedules' tickets, half-warps and levels end."""

import numpy as np
import pytest

from icsfoam_gb300 import cases

pytestmark = pytest.mark.gpu


def _open(binding, w, **over):
    h_cfg = cases.make_config(binding, w.settings, **over)
    from icsfoam_gb300 import abi

    h = abi.CaseHandle(binding, w.mesh, h_cfg)
    h.set_primitive(w.p, w.U, w.T)
    h.residual()
    h.assemble_jacobian()
    return h


SHAPES = {
    # levels of at most 31 / 32 / 33 rows: one short, one full and two tickets
    "levels_31": lambda: cases.bump_channel(31, 31, 1, ordering_mode="natural", second_order=False),
    "levels_32": lambda: cases.bump_channel(32, 32, 1, ordering_mode="natural", second_order=False),
    "levels_33": lambda: cases.bump_channel(33, 33, 1, ordering_mode="natural", second_order=False),
    "box_rcm_5": lambda: cases.random_box(5, ordering_mode="rcm"),
    "box_rcm_11": lambda: cases.random_box(11, ordering_mode="rcm"),
    # chains: fewer rows than chunks, one row per chunk, a short last chunk
    "chain_3": lambda: cases.shock_tube(3),
    "chain_37": lambda: cases.shock_tube(37),
    "chain_128": lambda: cases.shock_tube(128),
    "chain_129": lambda: cases.shock_tube(129),
    "chain_1000": lambda: cases.shock_tube(1000),
    # two colours on a few cells: level launches and the fused operator
    "two_colours_2x2x1": lambda: cases.bump_channel(2, 2, 1, ordering_mode="colour", second_order=False),
    "two_colours_9x5x3": lambda: cases.bump_channel(9, 5, 3, ordering_mode="colour", second_order=False),
}


# FP64: a row is a few dozen products, and round-off grows by at most the
# number of levels (< 70) along the sweep: 70 * 100 * 2^-53 < 1e-12.  Mixed:
# the same count in FP32 units, 70 * 100 * 2^-24 = 4e-4 at worst; the sweeps
# contract, so the rounding of a handful of levels (1e-5) bounds it.
@pytest.mark.parametrize("precision,tol", [(0, 1e-12), (1, 1e-5)])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_sweeps_follow_the_sequential_oracle(oracle_binding, gpu_binding, shape, precision, tol):
    w = SHAPES[shape]()
    hg, ho = _open(gpu_binding, w, precision=precision), _open(oracle_binding, w)
    r = np.random.default_rng(5).standard_normal((w.mesh.n_cells, 5))
    a, b = hg.precondition(r), ho.precondition(r)
    assert np.abs(a - b).max() <= tol * np.abs(b).max()
