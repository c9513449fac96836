"""The mixed form's FP64 reciprocal and square root (csrc/physics.cuh approx_rcp, approx_sqrt) against IEEE
division and square root: within one unit in the last place over the exponent range, and 1/0, 1/infinity,
sqrt(0), sqrt(infinity), negative and NaN arguments as IEEE gives them. The functions are device code without an
entry point of their own, so the test compiles a kernel of them."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from compas_b200 import build

pytestmark = pytest.mark.gpu

SRC = r"""
#include "physics.cuh"
__global__ void eval(const double* x, double* r, double* s, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    r[i] = compas::approx_rcp(x[i]);
    s[i] = compas::approx_sqrt(x[i]);
}
extern "C" int run(const double* x, double* r, double* s, int n) {
    eval<<<(n + 255) / 256, 256>>>(x, r, s, n);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? (int)cudaDeviceSynchronize() : (int)e;
}
"""


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not found")
    import torch

    d = tmp_path_factory.mktemp("quotients")
    src, out = os.path.join(d, "q.cu"), os.path.join(d, "q.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.check_call(["nvcc"] + build.ARCH + build.FLAGS + ["-I" + build.CSRC, "-shared", "-o", out, src])
    lib = ctypes.CDLL(out)

    def run(x):
        dev = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        r, s = torch.empty_like(dev), torch.empty_like(dev)
        torch.cuda.synchronize()
        assert lib.run(ctypes.c_void_p(dev.data_ptr()), ctypes.c_void_p(r.data_ptr()), ctypes.c_void_p(s.data_ptr()), len(x)) == 0
        return r.cpu().numpy(), s.cpu().numpy()

    return run


def test_within_one_unit_in_the_last_place(evaluate):
    rng = np.random.default_rng(0)
    x = rng.uniform(1.0, 2.0, 1 << 20) * 2.0 ** rng.integers(-1000, 1000, 1 << 20)
    edge = np.concatenate([np.nextafter(2.0 ** np.arange(-1000, 1000), 0.0), 2.0 ** np.arange(-1000, 1000.0)])
    x = np.concatenate([x, edge])
    r, s = evaluate(x)
    for got, want in ((r, 1.0 / x), (s, np.sqrt(x))):
        ulps = np.abs(got - want) / np.spacing(want)
        print(f"largest difference {ulps.max():.2f} ulp, {np.mean(ulps > 0):.1e} of the arguments differ")
        assert ulps.max() <= 1.0
    r, _ = evaluate(-x)
    assert np.all(np.abs(r + 1.0 / x) <= np.spacing(1.0 / x))


def test_zero_infinity_nan_and_negative_arguments(evaluate):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -1.0, -1e-3])
    r, s = evaluate(x)
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(r[:5], 1.0 / x[:5])
        np.testing.assert_array_equal(np.signbit(r[:4]), np.signbit(1.0 / x[:4]))
        np.testing.assert_array_equal(s, np.sqrt(x))
    # subnormal arguments: the reciprocal reads them as 0, the square root returns them
    r, s = evaluate(np.array([5e-324, 1e-310, -1e-310]))
    np.testing.assert_array_equal(r, [np.inf, np.inf, -np.inf])
    assert np.all(s[:2] < 1e-300) and np.isnan(s[2])
