"""The quotient by a fixed divisor of the panel kernels (csrc/fast_div.h),
compiled for the host: exact at both ends of every column of panels of any
height, below 2^21 entries (where the FP32 estimate alone is exact) and up to
2^30."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lowrankintegrators.jl_gb300", "csrc")
SOURCE = """
#include "fast_div.h"
extern "C" void quotients(int d, int count, const int* e, int* q) {
  const lri::wide::FastDiv by(d);
  for (int i = 0; i < count; ++i) q[i] = by.div(e[i]);
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("fast_div")
    (d / "q.cpp").write_text(SOURCE)
    subprocess.run([gxx, "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, str(d / "q.cpp"), "-o",
                    str(d / "q.so")], check=True)
    f = ctypes.CDLL(str(d / "q.so")).quotients

    def run(div, e):
        e = np.ascontiguousarray(e, np.int32)
        q = np.empty_like(e)
        p = ctypes.POINTER(ctypes.c_int)
        f(int(div), len(e), e.ctypes.data_as(p), q.ctypes.data_as(p))
        return q

    return run


@pytest.mark.parametrize("heights", [range(1, 4000), [32767, 32768], [114050, 107744, 102581, 105120, 205162, 228035],
                                     [10 ** 6 + 3, 4194303, 16777216, 16777217]])
def test_column_ends(quotients, heights):
    for n in heights:
        w = min(64, (1 << 30) // n)
        k = np.arange(w + 1, dtype=np.int64) * n
        e = np.unique(np.concatenate([k, k - 1, k + 1, k + n // 2]))
        e = e[(e >= 0) & (e < w * n)]
        assert np.array_equal(quotients(n, e), e // n), n


def test_random_entries(quotients):
    g = np.random.default_rng(2)
    for _ in range(300):
        w = int(g.integers(1, 65))
        n = int(np.exp(g.uniform(0.0, np.log((1 << 30) / w))))
        e = g.integers(0, max(1, n * w), 2000)
        assert np.array_equal(quotients(n, e), e // n), (n, w)
