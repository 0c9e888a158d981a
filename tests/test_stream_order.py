"""Every copy and fill of a handle's memory is ordered on the handle's stream.

A handle's kernels run on a non-blocking stream, which does not wait for the
default one, and a copy from pageable memory may return before the data is on
the device: a copy to the device or a fill on the default stream can reach
memory that a kernel already reads."""

import glob
import os
import re
import threading

import numpy as np
import pytest

from icsfoam_gb300 import _build, abi, cases


def test_no_copy_to_the_device_on_the_default_stream():
    for path in glob.glob(os.path.join(_build.CSRC, "*.cu*")):
        text = open(path).read()
        for call in re.findall(r"cudaMemcpy\([^;]*;", text):
            assert "HostToDevice" not in call, (path, call)
        assert "cudaMemset(" not in text, path


@pytest.mark.gpu
def test_handles_created_side_by_side_equal_one_created_alone(gpu_binding):
    w = cases.bump_channel(61, 31, 29, ordering_mode="colour")
    p = w.p * (1 + 0.02 * np.random.default_rng(3).uniform(-1, 1, w.mesh.n_cells))

    def source():
        h = abi.CaseHandle(gpu_binding, w.mesh, cases.make_config(gpu_binding, w.settings))
        h.set_primitive(p, w.U, w.T)
        return h.residual()

    alone = source()
    out = [[] for _ in range(6)]

    def work(k):
        for _ in range(4):
            out[k].append(source())

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(out))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert [len(o) for o in out] == [4] * len(out)
    assert all(np.array_equal(alone, s) for o in out for s in o)
