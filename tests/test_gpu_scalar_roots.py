"""The FP64 square root and reciprocal of the panel QR's scalars (csrc/wide.cuh,
Newton steps from FP32 estimates) beside CUDA's own: at most one unit in the
last place off the correctly rounded values.  (The last Newton step's residual
is exact to one rounding, so the error is half a unit and a rounding.)"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "wide.cuh"
__global__ void scalars(const double* x, int count, double* root, double* inv) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    root[i] = lri::wide::root(x[i]);
    inv[i] = lri::wide::reciprocal(x[i]);
  }
}
extern "C" int run(const double* x, int count, double* root, double* inv) {
  scalars<<<64, 256>>>(x, count, root, inv);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def scalars(lri, tmp_path_factory):
    import __graft_entry__ as ge
    import torch
    build = ge.load_build_module()
    d = tmp_path_factory.mktemp("scalars")
    (d / "s.cu").write_text(SOURCE)
    subprocess.run([build._nvcc(), *build.ARCH_FLAGS, *build.COMMON_FLAGS, "-Xcompiler", "-fvisibility=default",
                    "-I", build.CSRC, "-shared", "-cudart", "shared", str(d / "s.cu"), "-o", str(d / "s.so")], check=True)
    f = ctypes.CDLL(str(d / "s.so")).run

    def run(x):
        t = torch.from_numpy(x).cuda()
        out = torch.empty((2, len(x)), dtype=torch.float64, device="cuda")
        p = lambda a: ctypes.c_void_p(a.data_ptr())
        assert f(p(t), len(x), p(out[0]), p(out[1])) == 0
        return out.cpu().numpy()

    return run


def ulps(a, b):
    return np.abs(a.view(np.int64) - b.view(np.int64)).max()


@pytest.mark.parametrize("low,high", [(-0.01, 0.01), (-8, 8), (-29.9, 29.9)])
def test_roots_and_reciprocals(scalars, low, high):
    """1e-30 < x < 1e30, the range in which both take the Newton form."""
    g = np.random.default_rng(7)
    x = 10.0 ** g.uniform(low, high, 1 << 20)
    x[:4096] = 2.0 ** g.integers(int(np.ceil(low * 3.3)), int(high * 3.3) + 1, 4096)
    root, inv = scalars(x)
    assert ulps(root, np.sqrt(x)) <= 1
    assert ulps(inv, 1.0 / x) <= 1


def test_root_outside_the_newton_range(scalars):
    x = np.concatenate([10.0 ** np.random.default_rng(8).uniform(-307, -31, 4096),
                        10.0 ** np.random.default_rng(9).uniform(31, 307, 4096), [0.0, 5e-324, np.inf]])
    assert np.array_equal(scalars(x)[0], np.sqrt(x))
