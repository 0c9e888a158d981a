"""The FP32 runs of the Gram-Schmidt columns' sums, by the rules of k_column.cu:
a thread joins runs with their rounding errors kept (TwoSum), and no run holds
more products than a thread of one grid-stride launch per step over 608 blocks
of 256 threads adds in FP32, so no sum is rounded more than there."""

import os
import re

import numpy as np

from icsfoam_gb300 import _build

SOURCE = open(os.path.join(_build.CSRC, "k_column.cu")).read()


def _constant(pattern):
    return re.search(pattern, SOURCE).group(1)


def test_runs_are_no_longer_than_one_thread_s_share_of_a_launch():
    run_of = _constant(r"constexpr int RUN = ([^;]*);")
    run_of = eval("lambda U: " + re.sub(r"(.*)\?(.*):(.*)", r"(\2) if (\1) else (\3)", run_of).replace("/", "//"))
    small_grid = int(_constant(r"SMALL_GRID = (\d+)"))
    large = int(_constant(r"sizeof\(TV\) == 4 \? (\d+) :"))
    most = 151
    for n in np.unique(np.geomspace(5, 5.5e6, 4000).astype(int)):
        nv = -(-n // 4)
        G = max(1, min(most if n > large else min(most, small_grid), (nv + 127) // 128))
        chunks = -(-nv // G)
        U = next((u for u in range(2, 20, 2) if chunks <= 512 * u), None)
        if U is not None:  # longer slices: runs of at most eight chunks, as there from 5.6M entries on
            assert run_of(U) <= -(-nv // (608 * 256)), (n, U)


def test_joined_runs_keep_what_a_single_run_loses():
    f = np.float32
    rng = np.random.default_rng(0)
    runs = (1 + 1e-3 * rng.standard_normal((18, 4096))).astype(f)
    hi, lo, plain = runs[0].copy(), np.zeros(4096, f), runs[0].copy()
    for r in runs[1:]:
        s = hi + r
        b = s - hi
        lo = lo + ((hi - (s - b)) + (r - b))
        hi = s
        plain = plain + r
    exact = runs.astype(np.float64).sum(axis=0)
    # the joined sum's error is that of its lower part: 18 roundings at 2^-24 of 18 2^-24
    assert (np.abs(hi.astype(np.float64) + lo - exact) <= 18 * 18 * 2.0 ** -48).all()
    assert np.abs(plain - exact).max() > 1e-6
