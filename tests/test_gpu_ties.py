"""The reverse product is the transpose of the forward one where branches tie:
flows that are uniform or linear in space on uniform cells, with no cell
perturbed, put the limiters' ratios and the sides' sound speeds within rounding
of their switches in every cell (Venkatakrishnan's cap lies at r = 2, minmod's
at r = 1, the ratios of a linear profile), so both products have to decide each
branch on the same bits."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases, ordering
from icsfoam_gb300 import mesh as M

from test_gpu_diff import direction  # noqa: E402

pytestmark = pytest.mark.gpu

PROFILES = {
    "uniform": lambda x: (1.0, 1.0, [0.31, 0.17, -0.11]),
    "linear_T": lambda x: (1.0, 1.0 + 0.1 * x[:, 0], [0.31, 0.17, -0.11]),
    "linear": lambda x: (1.0 + 0.1 * x[:, 0] + 0.03 * x[:, 1], 1.0 + 0.05 * x[:, 0] - 0.02 * x[:, 2],
                         [0.31 + 0.1 * x[:, 0], 0.17 + 0.1 * x[:, 1], 0.2 * x[:, 0]]),
}


def _open(b, profile, flux, recon, n=(14, 6, 5), spacing=0.1):
    grid = np.stack(np.meshgrid(*[spacing * np.arange(k + 1) for k in n], indexing="ij"), axis=-1)
    free, slip = M.Patch("ends", M.PATCH_ZERO_GRADIENT), M.Patch("sides", M.PATCH_SLIP)
    m = ordering.apply(M.hex_mesh(grid, {"xmin": free, "xmax": free, "ymin": slip, "ymax": slip, "zmin": slip,
                                         "zmax": slip}), "colour")
    w = cases.bump_channel(4, 4, 4, flux=flux)
    p, T, U = PROFILES[profile](m.C)
    one = np.ones(m.n_cells)
    h = abi.CaseHandle(b, m, cases.make_config(b, w.settings, recon_rho=recon, recon_U=recon, recon_T=recon))
    h.set_primitive(1e5 * p * one, np.stack([340.0 * c * one for c in U], axis=1), 300.0 * T * one)
    return h


# both sums are a few hundred products per entry in FP64: 1e-12 of |u| |J v| is
# a few thousand units of 2^-53, a branch that differs in one cell of a hundred
# leaves 1e-3
@pytest.mark.parametrize("profile", list(PROFILES))
@pytest.mark.parametrize("flux", ["HLLC", "AUSMPlusUp", "ROE"])
@pytest.mark.parametrize("recon", [1, 2, 3, 4])
def test_reverse_product_transposes_the_forward_one_at_ties(gpu_binding, profile, flux, recon):
    h = _open(gpu_binding, profile, flux, recon)
    W = h.get_state()["W"]
    rng = np.random.default_rng(8)
    for s in range(2):
        v = direction(W, 20 + s)
        u = rng.standard_normal(W.shape)
        Jv, JTu = h.jvp(v), h.vjp_recompute(u)
        lhs, rhs = float(np.sum(u * Jv)), float(np.sum(JTu * v))
        assert abs(lhs - rhs) <= 1e-12 * np.linalg.norm(u) * np.linalg.norm(Jv)
