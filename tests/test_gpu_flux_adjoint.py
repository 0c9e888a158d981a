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
