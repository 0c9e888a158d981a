"""The backward walks of the flux functions on every branch they have:
subsonic and supersonic faces of both directions, low Mach numbers, the
entropy fix, a moving frame."""

import numpy as np
import pytest

from icsfoam_gb300 import cases
from icsfoam_gb300 import mrf as MRF

from test_gpu_diff import _over, direction, open_case  # noqa: E402
from test_gpu_parity import perturb  # noqa: E402

pytestmark = pytest.mark.gpu


# <u, J v> = <J^T u, v>, J v by dual numbers through the flux functions and
# J^T u by the backward walks: both sums are a few hundred products per entry
# in FP64, so they agree to 1e-12 of |u| |J v| (a few thousand units of 2^-53)
def _transpose(h, W):
    rng = np.random.default_rng(8)
    for s in range(2):
        v = direction(W, 20 + s)
        u = rng.standard_normal(W.shape)
        Jv, JTu = h.jvp(v), h.vjp_recompute(u)
        lhs, rhs = float(np.sum(u * Jv)), float(np.sum(JTu * v))
        assert abs(lhs - rhs) <= 1e-12 * np.linalg.norm(u) * np.linalg.norm(Jv)


@pytest.mark.parametrize("mach", [0.02, 0.95, 2.5, -0.95, -2.5])
@pytest.mark.parametrize("flux", ["HLLC", "AUSMPlusUp", "ROE"])
def test_flux_adjoints_on_every_branch(gpu_binding, flux, mach):
    w = cases.bump_channel(11, 5, 3, mach=abs(mach), ordering_mode="colour", flux=flux)
    w.U = w.U * np.sign(mach)
    h = open_case(gpu_binding, _over(perturb(w), entropy_fix_coeff=0.3))
    _transpose(h, h.get_state()["W"])


@pytest.mark.parametrize("flux", ["HLLC", "AUSMPlusUp", "ROE"])
def test_flux_adjoints_in_a_moving_frame(gpu_binding, flux):
    w = perturb(cases.annular_sector(4, 6, 6, ordering_mode="colour", flux=flux, sides="slip"))
    h = open_case(gpu_binding, w)
    h.set_mrf(MRF.frame_fields(w.mesh, *w.mrf), 0)
    _transpose(h, h.get_state()["W"])


def test_vjp_before_and_after_the_exact_jacobian(gpu_binding):
    """ics_vjp serves a new state's first calls by the reverse chain: they equal
    the products with the assembled Jacobian (1e-10 of the largest entry, the
    bound of the two routes), and the Jacobian is there when it is asked for."""
    w = perturb(cases.bump_channel(9, 5, 3, ordering_mode="colour"))
    h = open_case(gpu_binding, w)
    u = np.random.default_rng(6).standard_normal((w.mesh.n_cells, 5))
    first = h.vjp(u)
    ptr, cols, blocks = h.get_exact_jacobian()
    rows = np.repeat(np.arange(w.mesh.n_cells), np.diff(ptr))
    dense = np.zeros((w.mesh.n_cells, 5))
    np.add.at(dense, cols, np.einsum("jik,ji->jk", blocks, u[rows]))
    scale = np.abs(dense).max(axis=0)
    assert (np.abs(first - dense) <= 1e-10 * scale).all()
    h.set_conservative(h.get_state()["W"])  # a new state: the count starts again
    calls = [h.vjp(u) for _ in range(18)]   # beyond the calls the reverse chain serves
    assert all((np.abs(c - dense) <= 1e-10 * scale).all() for c in calls)
    assert np.array_equal(calls[16], calls[17])
