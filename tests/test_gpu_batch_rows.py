"""Batched replicas whose rows, boxes and cell grids differ: from one particle to boxes of
one cell, of many cells and of grids too short for the unwrapped coordinates, at
every lanes-per-particle bound; and the FP32 root and reciprocals of the evaluators."""

import ctypes
import subprocess

import numpy as np
import pytest

import azplugins_gb300 as az

pytestmark = pytest.mark.gpu

# particles, density, r_cut (buffer 0.4)
REPLICAS = [
    (1, 0.01, 1.0),      # one cell (no candidates but the particle)
    (33, 0.3, 1.6),      # L 4.8, one cell
    (700, 0.5, 5.1),     # L 11.2 = 2.03 r_list: one cell, rows of 349 entries
    (1000, 0.8, 2.6),    # L 10.8: 3 cells
    (1331, 0.7, 1.9),    # L 12.4: 5 cells, the shortest grid without the second wrap
    (2744, 0.8, 4.5),    # L 15.1: 3 cells of 100 particles
    (2744, 0.8, 3.9),    # L 15.1: 3 cells
    (4097, 0.9, 1.1),    # L 16.6: 11 cells of a few particles
]


def _snaps(seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for n, rho, _ in REPLICAS:
        L = (n / rho) ** (1.0 / 3.0)
        m = int(np.ceil(round(n ** (1.0 / 3.0), 9)))
        g = (np.arange(m) + 0.5) * (L / m) - 0.5 * L
        x = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
        x = x[rng.permutation(len(x))[:n]] + rng.uniform(-0.1, 0.1, (n, 3)) * (L / m)
        s = az.Snapshot(n)
        s.particles.types = ["A"]
        s.particles.position = x - L * np.floor(x / L + 0.5)
        s.particles.velocity = rng.normal(size=(n, 3))
        s.particles.typeid = np.zeros(n, dtype=np.int32)
        s.particles.acceleration = np.zeros((n, 3))
        s.configuration.box = [L] * 3 + [0.0] * 3
        out.append(s)
    return out


@pytest.mark.parametrize("precision,tpp,block", [("fp64", 1, 256), ("fp64", 32, 64), ("fp32", 1, 256), ("fp32", 8, 512),
                                                 ("fp32", 32, 64), ("fp32", 16, 128)])
def test_accelerations_of_uneven_replicas(precision, tpp, block):
    from azplugins_gb300.batch import ReplicaBatch

    snaps = _snaps(7)
    eps, kappa, delta, gamma, dt = 1.0, 0.7, 0.3, 1.0, 0.001
    b = ReplicaBatch(snaps, az.pair.ExpandedYukawa, [dict(epsilon=eps, kappa=kappa, delta=delta)] * len(snaps),
                     [r[2] for r in REPLICAS], list(range(len(snaps))), dt=dt, kT=0.0, gamma=gamma,
                     precision=precision)
    b.set_tpp(tpp)
    b.set_block(block)
    b.run(1)
    arrays = b.get_arrays()
    for r, (n, _, rc) in enumerate(REPLICAS):
        x, v, a, _ = b.replica(r, arrays)
        L = snaps[r].configuration.box[0]
        f = np.zeros((n, 3))
        scale = np.zeros(n)
        for i0 in range(0, n, 256):
            d = x[i0:i0 + 256, None] - x[None]
            d -= L * np.rint(d / L)
            q = (d * d).sum(-1)
            rr = np.sqrt(np.where(q > 0, q, 1.0))
            s = rr - delta
            w = eps * np.exp(-kappa * s) / s * (kappa + 1.0 / s) / rr
            w = np.where((q > 0) & (q < rc * rc), w, 0.0)
            f[i0:i0 + 256] = (w[..., None] * d).sum(1)
            scale[i0:i0 + 256] = (w * rr).sum(1)
        # a = f - gamma v(t + dt / 2), and the v returned is that plus dt a / 2
        a_ref = (f - gamma * v) / (1.0 - 0.5 * gamma * dt)
        # FP32: fixed-point and component roundings of a pair (a few 2^-24 in r, times the
        # steepness of w, 2 + kappa r + 2 r / s < 16) against the sum of |f|; FP64 likewise
        u = 16.0 * (2.0 ** -22 if precision == "fp32" else 2.0 ** -51)
        tol = u * (scale + gamma * np.abs(v).max() + 1.0)
        assert (np.abs(a - a_ref).max(1) < tol).all(), r
    b.close()


def test_results_that_are_held_stay():
    from azplugins_gb300.batch import ReplicaBatch

    snaps = _snaps(8)[1:3]
    b = ReplicaBatch(snaps, az.pair.ExpandedYukawa, [dict(epsilon=1.0, kappa=1.0, delta=0.0)] * 2, [1.6, 2.0], [1, 2],
                     dt=0.001)
    held, copies = [], []
    for k in range(5):
        b.run(2)
        arrays = b.get_arrays()
        # whole sets, and a slice of one array whose set is dropped
        held.append(arrays if k % 2 else arrays[1][3:9, 1:])
        copies.append([np.array(x) for x in held[-1]] if k % 2 else np.array(held[-1]))
        del arrays
    for h, c in zip(held, copies):
        for x, y in zip(h, c):
            assert np.array_equal(x, y)
    first = b.get_arrays()
    assert all(np.array_equal(x, y) for x, y in zip(first, b.get_arrays()))
    b.close()


SRC = r"""
#include "fp32.cuh"
using namespace azp;
__global__ void k(const float* x, const float* a, float* out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float root, inv;
    f_root(x[i], root, inv);
    out[i] = f_rcp(x[i]);
    out[n + i] = root;
    out[2 * n + i] = inv;
    out[3 * n + i] = f_over(a[i], root, inv);
}
extern "C" __attribute__((visibility("default"))) int run(const float* x, const float* a, float* out, int n)
{
    k<<<(n + 127) / 128, 128>>>(x, a, out, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.mark.parametrize("lo,hi", [(-2, 2), (-40, 40), (-100, 100)])
def test_fp32_functions_are_rounded(tmp_path, lo, hi):
    import torch

    from azplugins_gb300 import build

    (tmp_path / "m.cu").write_text(SRC)
    so = str(tmp_path / "m.so")
    subprocess.run([build.nvcc(), "-shared", "-o", so, str(tmp_path / "m.cu"), "-I", build.CSRC]
                   + build.common_flags(), check=True, capture_output=True)
    rng = np.random.Generator(np.random.PCG64(9))
    n = 300000
    x = (rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(lo, hi, n)).astype(np.float32)
    a = (rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-4, 5, n)).astype(np.float32)
    xd, ad = torch.from_numpy(x).cuda(), torch.from_numpy(a).cuda()
    out = torch.empty((4, n), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(t.data_ptr()) for t in (xd, ad, out)]
    assert ctypes.CDLL(so).run(*p, n) == 0
    o = out.cpu().numpy()
    x64, root64 = x.astype(np.float64), o[1].astype(np.float64)
    for got, ref in ((o[0], 1.0 / x64), (o[1], np.sqrt(x64)), (o[2], 1.0 / root64), (o[3], a.astype(np.float64) / root64)):
        ulp = np.spacing(np.abs(ref).astype(np.float32)).astype(np.float64)
        # the rounding of the last FMA, and the seed's squared error (2^-22) squared once more
        assert (np.abs(got - ref) <= 0.501 * ulp).all()
