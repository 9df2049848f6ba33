"""Rounding of the FP64 reciprocal, root and quotient of the evaluators: as the operators
round, also for quotients of very small and very large numbers."""

import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include "evaluators.cuh"
using namespace azp;
__global__ void k64(const double* x, const double* a, double* out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = rcp(x[i]);
    out[n + i] = root(x[i]);
    out[2 * n + i] = over(a[i], x[i]);
}
extern "C" __attribute__((visibility("default"))) int run64(const double* x, const double* a, double* out, int n)
{
    k64<<<(n + 127) / 128, 128>>>(x, a, out, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def module(tmp_path_factory):
    from azplugins_gb300 import build

    d = tmp_path_factory.mktemp("limits")
    (d / "m.cu").write_text(SRC)
    so = str(d / "m.so")
    subprocess.run([build.nvcc(), "-shared", "-o", so, str(d / "m.cu"), "-I", build.CSRC] + build.common_flags(),
                   check=True, capture_output=True)
    return ctypes.CDLL(so)


def _run(module, x, a, rows):
    import torch

    xd, ad = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x, a))
    out = torch.empty((rows, len(x)), dtype=xd.dtype, device="cuda")
    torch.cuda.synchronize()
    assert module.run64(ctypes.c_void_p(xd.data_ptr()), ctypes.c_void_p(ad.data_ptr()), ctypes.c_void_p(out.data_ptr()), len(x)) == 0
    return out.cpu().numpy()


def test_fp64_quotients_at_the_ends(module):
    x = np.array([3.0, 3.0, 7.0, 0.0, np.inf, 3.0, np.nan, 1e-320, 1e300, 3.0])
    a = np.array([1e-320, 1e-290, 1e306, 2.0, 2.0, np.inf, 1.0, 1e-310, 1e-300, 0.0])
    with np.errstate(all="ignore"):
        ref = a / x
    np.testing.assert_allclose(_run(module, x, a, 3)[2], ref, rtol=2.0 ** -52, atol=5e-324, equal_nan=True)


def test_fp64_forms_are_rounded_as_the_operators(module):
    rng = np.random.Generator(np.random.PCG64(8))
    n = 2000000
    x = rng.uniform(1.0, 4.0, n) * 2.0 ** rng.integers(-8, 8, n)
    a = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-40, 40, n)
    r = _run(module, x, a, 3)
    for got, want in zip(r, (1.0 / x, np.sqrt(x), a / x)):
        # one rounding of a value known to 2^-8 ulp or better (a seed of 2^-21 cubed; the
        # residual of a reciprocal's last place): a neighbour at most, in 1 of 100 at most
        assert np.abs((got - want) / np.spacing(want)).max() <= 1.0
        assert (got != want).mean() < 0.01
