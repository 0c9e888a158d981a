"""The route of ics_vjp is the caller's: every call at a state gives the same
bits at the same cost until the program assembles the exact Jacobian, and the
assembled one is used from there until the state changes."""

import numpy as np
import pytest

from icsfoam_gb300 import cases

from test_gpu_diff import open_case  # noqa: E402
from test_gpu_parity import perturb  # noqa: E402

pytestmark = pytest.mark.gpu


def test_equal_calls_give_equal_bits_until_the_jacobian_is_assembled(gpu_binding):
    w = perturb(cases.bump_channel(9, 5, 3, ordering_mode="colour"))
    h = open_case(gpu_binding, w)
    u = np.random.default_rng(6).standard_normal((w.mesh.n_cells, 5))
    calls, launches = [], []
    for _ in range(40):
        before = h.launch_count()
        calls.append(h.vjp(u))
        launches.append(h.launch_count() - before)
    assert all(np.array_equal(c, calls[0]) for c in calls)
    assert len(set(launches)) == 1
    assert np.array_equal(calls[0], h.vjp_recompute(u))
    h.assemble_exact_jacobian()
    assembled = [h.vjp(u) for _ in range(3)]
    assert all(np.array_equal(a, assembled[0]) for a in assembled)
    # the products of one Jacobian by two routes: 1e-10 of the largest entry
    scale = np.abs(assembled[0]).max(axis=0)
    assert (np.abs(calls[0] - assembled[0]) <= 1e-10 * scale).all()
    h.set_conservative(h.get_state()["W"])  # a new state
    assert np.array_equal(h.vjp(u), h.vjp_recompute(u))


def test_the_blocks_are_there_after_a_product(gpu_binding):
    w = perturb(cases.bump_channel(9, 5, 3, ordering_mode="colour"))
    a, b = open_case(gpu_binding, w), open_case(gpu_binding, w)
    u = np.random.default_rng(6).standard_normal((w.mesh.n_cells, 5))
    a.vjp(u)
    b.assemble_exact_jacobian()
    assert np.array_equal(a.get_exact_jacobian()[2], b.get_exact_jacobian()[2])
    assert np.array_equal(a.vjp(u), b.vjp(u))  # both hold the assembled one now
