"""The viscous terms of a cell are summed on their own: beside a pressure a
hundred thousand times larger they keep their digits."""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases, ordering
from icsfoam_gb300 import mesh as M

pytestmark = pytest.mark.gpu


# A shear flow u(y) = a y^2 at uniform pressure and temperature on cells of edge
# 2^-3: the pressure forces of a cell cancel exactly, so its x momentum residual
# is the viscous force mu h (u_{j+1} - 2 u_j + u_{j-1}).  A face term is up to
# 20 times the force and carries a few roundings of 2^-53, which makes 1e-13 of
# the force; rounded beside p S it would be off by 1e-5 of it.
@pytest.mark.parametrize("flux", [0, 1])  # AUSM+up, HLLC
def test_viscous_force_beside_a_large_pressure(gpu_binding, oracle_binding, flux):
    h, a, n = 0.125, 1.0, (5, 10, 4)
    grid = np.stack(np.meshgrid(*[h * np.arange(k + 1) for k in n], indexing="ij"), axis=-1)
    end = M.Patch("sides", M.PATCH_ZERO_GRADIENT)
    m = ordering.apply(M.hex_mesh(grid, {s: end for s in ("xmin", "xmax", "ymin", "ymax", "zmin", "zmax")}), "colour")
    settings = dict(cases.random_box(4).settings, flux_scheme=flux, sutherland=0, mu=1.8e-5)
    N, y = m.n_cells, m.C[:, 1]
    inner = ((m.C > 1.1 * h) & (m.C < (np.array(n) - 1.1) * h)).all(axis=1) & (np.abs(y - 0.5 * n[1] * h) < 3.1 * h)
    assert inner.sum() >= 12
    for b in (gpu_binding, oracle_binding):
        cfg = cases.make_config(b, settings)
        assert cfg.viscous and not cfg.sutherland
        c = abi.CaseHandle(b, m, cfg)
        c.set_primitive(np.full(N, 131072.0), np.stack([a * y * y, 0 * y, 0 * y], axis=1), np.full(N, 300.0))
        force = c.residual()[inner, 1]
        expect = cfg.mu * h * 2 * a * h * h
        assert np.abs(force - expect).max() <= 1e-11 * expect, (np.abs(force - expect).max() / expect)
