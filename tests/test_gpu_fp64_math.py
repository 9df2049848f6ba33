"""The FP64 reciprocal and square roots of csrc/fp64.cuh against correctly rounded
results: a small module built from the header evaluates them on the GPU."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include "fp64.cuh"
using namespace azp;
__global__ void k(const double* x, double* out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = d_rcp(x[i]);
    out[n + i] = d_rsqrt(x[i]);
    out[2 * n + i] = d_sqrt(x[i]);
    out[3 * n + i] = less_nonneg(fabs(x[i]), 2.0) ? 1.0 : 0.0;
    out[4 * n + i] = magnitude_above(x[i], 2.0) ? 1.0 : 0.0;
}
extern "C" __attribute__((visibility("default"))) int run(const double* x, double* out, int n)
{
    k<<<(n + 127) / 128, 128>>>(x, out, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def module(tmp_path_factory):
    from azplugins_gb300 import build

    d = tmp_path_factory.mktemp("fp64")
    (d / "m.cu").write_text(SRC)
    so = str(d / "m.so")
    subprocess.run([build.nvcc(), "-shared", "-o", so, str(d / "m.cu"), "-I", build.CSRC] + build.common_flags(),
                   check=True, capture_output=True)
    return ctypes.CDLL(so)


def _run(module, x):
    import torch

    xd = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    out = torch.empty((5, len(x)), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert module.run(ctypes.c_void_p(xd.data_ptr()), ctypes.c_void_p(out.data_ptr()), len(x)) == 0
    return out.cpu().numpy()


@pytest.mark.parametrize("lo,hi", [(-2, 2), (-30, 30), (-99, 99), (-320, 320)])
def test_refined_functions_round_to_an_ulp(module, lo, hi):
    rng = np.random.Generator(np.random.PCG64(5 + hi))
    x = rng.uniform(1.0, 2.0, size=200000) * 2.0 ** rng.integers(lo, hi, size=200000)
    # the ends of the seeds' range and exact powers of two among them
    x[:8] = [1.0, 2.0, 0.5, 4.0, np.nextafter(1.0, 0.0), np.nextafter(2.0, 4.0), 2.0 ** lo, np.nextafter(2.0 ** hi, 0.0)]
    r = _run(module, x)
    # one rounding of the last operation plus the residual of the iteration: 1 ulp;
    # 1 / sqrt adds the rounding of x y and of its correction: 2 ulp
    assert np.abs((r[0] - 1.0 / x) / np.spacing(1.0 / x)).max() <= 1.0
    assert np.abs((r[1] - 1.0 / np.sqrt(x)) / np.spacing(1.0 / np.sqrt(x))).max() <= 2.0
    assert np.abs((r[2] - np.sqrt(x)) / np.spacing(np.sqrt(x))).max() <= 1.0
    n = _run(module, -x)
    assert np.array_equal(n[0], -r[0])


def test_special_values(module):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -1.0, 5e-324, 1e-310, 1.7e308, 2.0, np.nextafter(2.0, 0.0), -2.0,
                  -3.0])
    r = _run(module, x)
    with np.errstate(all="ignore"):
        assert np.array_equal(r[0], 1.0 / x, equal_nan=True)
        assert np.array_equal(r[2], np.sqrt(x), equal_nan=True)
        ref = 1.0 / np.sqrt(x)
    assert np.allclose(r[1], ref, rtol=1e-15, atol=0.0, equal_nan=True)
    with np.errstate(invalid="ignore"):
        assert np.array_equal(r[3] == 1.0, np.abs(x) < 2.0)
        assert np.array_equal((r[4] == 1.0)[~np.isnan(x)], (np.abs(x) > 2.0)[~np.isnan(x)])
