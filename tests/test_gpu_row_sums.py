"""Rounding of the FP64 products and sweeps: against sums in extended precision
of the same blocks, the device's error is no larger than that of plain FP64
sums that form each block product before they add it to the row.  (Terms added
one by one to the row's sum round at the size of its diagonal part: 1.5 times
the error.)"""

import numpy as np
import pytest

from icsfoam_gb300 import abi, cases

from test_gpu_parity import perturb  # noqa: E402

pytestmark = pytest.mark.gpu


def _sums(m, J, dtype):
    diag, low, up = (np.asarray(a, dtype) for a in J)
    own, nei = m.owner, m.neighbour
    second = np.zeros(m.n_cells, bool)  # two colours: no face joins cells of one
    second[nei] = True

    def mv(M, x):
        return sum(M[:, :, k] * x[:, k, None] for k in range(5))

    def product(x):
        y = mv(diag, x)
        np.add.at(y, own, mv(up, x[nei]))
        np.add.at(y, nei, mv(low, x[own]))
        return y

    def sweeps(r):
        rD = (1.0 / np.abs(np.einsum("nii->ni", J[0])).max(axis=1)).astype(dtype)[:, None]
        f = r.copy()
        np.add.at(f, nei, -mv(low, (rD * r)[own]))
        z = np.where(second[:, None], rD * f, dtype(0))
        t = f.copy()
        np.add.at(t, own, -mv(up, z[nei]))
        return np.where(second[:, None], z, rD * t)

    return product, sweeps


# rows on five lanes each, and a row per thread; 1.1: the scatter of the mean
# square over 10^4 rounding errors is 2%
@pytest.mark.parametrize("shape", [(25, 13, 9), (61, 33, 31)])
def test_products_and_sweeps_round_as_plain_sums(gpu_binding, shape):
    w = perturb(cases.bump_channel(*shape, ordering_mode="colour"))
    h = abi.CaseHandle(gpu_binding, w.mesh, cases.make_config(gpu_binding, w.settings))
    h.set_primitive(w.p, w.U, w.T)
    h.set_pseudo_co(np.full(w.mesh.n_cells, 200.0))
    h.residual()
    h.assemble_jacobian()
    J = h.get_jacobian()
    W = h.get_state()["W"]
    x = W * (1 + 1e-2 * np.sin(3 * w.mesh.C[:, :1]))
    exact, plain = _sums(w.mesh, J, np.longdouble), _sums(w.mesh, J, np.float64)
    r = plain[0](x)
    for k, (device, v) in enumerate(((h.matrix_mul, x), (h.precondition, r))):
        e = exact[k](v.astype(np.longdouble))
        scale = np.sqrt((e ** 2).mean(axis=0))
        rms = [np.sqrt((((np.asarray(a, np.longdouble) - e) / scale) ** 2).mean()) for a in (device(v), plain[k](v))]
        assert rms[0] <= 1.1 * rms[1], rms


def _cell_by_cell(m, J, dtype):
    """Both sweeps row after row, in the order of the cells."""
    diag, low, up = (np.asarray(a, dtype) for a in J)
    rD = (1.0 / np.abs(np.einsum("nii->ni", J[0])).max(axis=1)).astype(dtype)
    below, above = [[] for _ in range(m.n_cells)], [[] for _ in range(m.n_cells)]
    for f, (o, n) in enumerate(zip(m.owner, m.neighbour)):
        above[o].append((n, up[f]))
        below[n].append((o, low[f]))

    def sweeps(r):
        x = r.copy()
        for c in range(m.n_cells):
            for j, B in below[c]:
                x[c] = x[c] - (B * (rD[j] * x[j])).sum(axis=1)
        for c in reversed(range(m.n_cells)):
            for j, B in above[c]:
                x[c] = x[c] - (B * x[j]).sum(axis=1)
            x[c] = rD[c] * x[c]
        return x

    return sweeps


# the scan of a chain of many levels and the sync-free sweeps; 1.2: a few
# thousand rounding errors, correlated along the levels
@pytest.mark.parametrize("shape", ["chain_129", "chain_1000", "levels"])
def test_sweeps_of_many_levels_round_as_plain_ones(gpu_binding, shape):
    w = {"chain_129": lambda: cases.shock_tube(129), "chain_1000": lambda: cases.shock_tube(1000),
         "levels": lambda: cases.bump_channel(19, 9, 7, ordering_mode="natural")}[shape]()
    w = perturb(w)
    h = abi.CaseHandle(gpu_binding, w.mesh, cases.make_config(gpu_binding, w.settings))
    h.set_primitive(w.p, w.U, w.T)
    h.begin_time_step()
    h.residual()
    h.assemble_jacobian()
    J = h.get_jacobian()
    errors = np.zeros(2)
    for seed in range(4):
        r = np.random.default_rng(seed).standard_normal((w.mesh.n_cells, 5)) * np.abs(h.get_state()["W"]).max(axis=0)
        e = _cell_by_cell(w.mesh, J, np.longdouble)(r.astype(np.longdouble))
        scale = np.maximum(np.sqrt((e ** 2).mean(axis=0)), 1e-300)
        for k, a in enumerate((h.precondition(r), _cell_by_cell(w.mesh, J, np.float64)(r))):
            errors[k] += float((((np.asarray(a, np.longdouble) - e) / scale) ** 2).mean())
    assert np.sqrt(errors[0]) <= 1.2 * np.sqrt(errors[1]), np.sqrt(errors)
