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
