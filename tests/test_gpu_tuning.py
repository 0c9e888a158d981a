"""The autotuner times a choice only where its candidates run different kernels."""

import pytest

from icsfoam_gb300 import cases

from test_gpu_diff import open_case  # noqa: E402

pytestmark = pytest.mark.gpu


# sync-free sweeps, the chain scan, and two levels of few FP64 rows: the reverse
# sweep's rows per thread choose nothing there
@pytest.mark.parametrize("n", range(5))
@pytest.mark.parametrize("shape", ["levels", "chain", "few_rows"])
def test_rows_per_thread_stay_where_they_choose_nothing(gpu_binding, shape, n):
    w = {"levels": lambda: cases.bump_channel(14 + n, 7, 5, ordering_mode="natural"),
         "chain": lambda: cases.shock_tube(300 + n),
         "few_rows": lambda: cases.bump_channel(14 + n, 7, 5, ordering_mode="colour")}[shape]()
    h = open_case(gpu_binding, w)
    h.residual()
    h.assemble_jacobian()
    t = h.autotune()
    assert t["reverse_rows"] == 1 and t["mgs_blocks"] == 608 and not t["from_cache"]
