"""The f64 helpers of the kernels against exact values and against CUDA's own
rsqrt and division. They are inline device functions, so a small library is
built around their header."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

from solarsystemsimulator_b200 import build as sss_build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "sss_internal.cuh"
__global__ void k(const double* x, long long n, double* out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double d = x[i], v = rsqrt(d);
    out[i] = sss_gm_rinv3(1.0, d);
    out[n + i] = (v * v) * v;
    out[2 * n + i] = sss_recip_f64(d);
    out[3 * n + i] = 1.0 / d;
}
extern "C" int run(const double* x, long long n, double* out) {
    k<<<(unsigned)((n + 255) / 256), 256>>>(x, n, out);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    d = tmp_path_factory.mktemp("math")
    src, lib = str(d / "math.cu"), str(d / "libmath.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([sss_build._nvcc(), *sss_build.ARCH_FLAGS, *sss_build.NVCC_FLAGS, f"-I{sss_build.INCLUDE}",
                    f"-I{sss_build.CSRC}", "-o", lib, src], check=True, capture_output=True)
    run = ctypes.CDLL(lib).run
    run.argtypes = [ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p]

    def call(x):
        t = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        out = torch.empty((4, len(x)), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert run(t.data_ptr(), len(x), out.data_ptr()) == 0
        return out.cpu().numpy()

    assert os.path.exists(lib)
    return call


def test_series_of_the_pair_factor(evaluate):
    """r^-3 from r^2 over 128 binades. The square of the seed is rounded once,
    which moves the result by half of that, the cube and the sum once each:
    2.5 x 2^-53, and 1.5e-17 for the terms left out. No further off than the
    cube of CUDA's rsqrt, at most and on average."""
    rng = np.random.default_rng(0)
    r2 = rng.uniform(1.0, 2.0, 1 << 20) * 2.0 ** rng.integers(-64, 64, 1 << 20)
    got = evaluate(r2)
    x = r2.astype(np.longdouble)
    exact = 1.0 / (x * np.sqrt(x))
    err = [np.abs((g - exact) / exact).astype(np.float64) for g in got[:2]]
    assert err[0].max() <= 2.5 * 2.0 ** -53 + 1.5e-17
    assert err[0].max() <= err[1].max() and (err[0] ** 2).mean() <= (err[1] ** 2).mean()


def test_pair_factor_of_special_values(evaluate):
    got = evaluate(np.array([np.inf, np.nan, 1e300, 1e-200]))
    assert got[0][0] == 0.0 and np.isnan(got[0][1]) and got[0][2] == 0.0
    assert abs(got[0][3] / 1e300 - 1.0) < 1e-15


def test_reciprocal(evaluate):
    """1 / d over 128 binades: the last step rounds once, its argument's error
    is squared away (below 2^-14 twice): 2^-53, and CUDA's quotient or a
    neighbour of it."""
    rng = np.random.default_rng(1)
    d = rng.uniform(1.0, 2.0, 1 << 20) * 2.0 ** rng.integers(-64, 64, 1 << 20)
    got = evaluate(d)
    exact = 1.0 / d.astype(np.longdouble)
    assert np.abs((got[2] - exact) / exact).max() <= 1.01 * 2.0 ** -53
    assert np.abs(got[2].view(np.int64) - got[3].view(np.int64)).max() <= 1
