"""ExpandedYukawa in FP32 where r or r - delta is zero, as the operators have it; energies of
coincident particles."""

import ctypes
import subprocess

import numpy as np
import pytest

import azplugins_gb300 as az

pytestmark = pytest.mark.gpu

SRC = r"""
#include "evaluators.cuh"
using namespace azp;
__global__ void k32(const float* x, const float* a, float* out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // ExpandedYukawa with epsilon 2, kappa 1.5, delta a
    const float rec[PAIR_REC] = {2.0f, 1.5f, a[i], 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    ExpandedYukawa::eval(rec, x[i], out[i], out[n + i]);
}
extern "C" __attribute__((visibility("default"))) int run32(const float* x, const float* a, float* out, int n)
{
    k32<<<(n + 127) / 128, 128>>>(x, a, out, n);
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
    assert module.run32(ctypes.c_void_p(xd.data_ptr()), ctypes.c_void_p(ad.data_ptr()), ctypes.c_void_p(out.data_ptr()), len(x)) == 0
    return out.cpu().numpy()


def test_yukawa_where_r_or_r_minus_delta_is_zero(module):
    # coincident particles, a pair exactly delta apart, and ordinary ones
    x = np.array([0.0, 0.0, 0.0, 0.25, 1.0, 4.0], dtype=np.float32)
    delta = np.array([0.3, -0.3, 0.0, 0.5, 0.3, 0.3], dtype=np.float32)
    f, u = _run(module, x, delta, 2)
    with np.errstate(all="ignore"):
        r = np.sqrt(x)
        s = r - delta
        uu = 2 * np.exp(np.float32(-1.5) * s) / s
        ff = uu * (np.float32(1.5) + 1 / s) / r
    np.testing.assert_allclose(u, uu, rtol=1e-6)
    np.testing.assert_allclose(f, ff, rtol=1e-6)


def test_energies_of_coincident_particles_fp32(orc):
    """ExpandedYukawa at r = 0: the energy is finite."""
    from azplugins_gb300 import _engine

    eps, kappa, delta = 2.0, 1.5, 0.3
    snap = az.Snapshot(4)
    snap.particles.position = np.array([[1.0, 2.0, 0.5]] * 2 + [[-3.0, -3.0, 3.0], [-2.0, -3.0, 3.0]])
    snap.particles.acceleration = np.zeros((4, 3))
    snap.configuration.box = [12.0] * 3 + [0.0] * 3
    y = az.pair.ExpandedYukawa(nlist=az.nlist.Cell(buffer=0.3), default_r_cut=2.5)
    y.params[("A", "A")] = dict(epsilon=eps, kappa=kappa, delta=delta)
    sim = az.Simulation(seed=1, precision="fp32")
    sim.create_state_from_snapshot(snap)
    integ = az.md.Integrator(dt=0.005, methods=[az.methods.LangevinFlow("all", kT=1.0,
                                                flow_field=az.flow.ConstantFlow((0.0, 0.0, 0.0)))], forces=[y])
    u = [eps * np.exp(-kappa * (r - delta)) / (r - delta) for r in (0.0, 1.0)]
    want = 0.5 * np.array([u[0], u[0], u[1], u[1]])
    eng = _engine.Engine(sim, integ, snap)
    eng.push(snap, 0)
    np.testing.assert_allclose(eng.forces()[0][:, 3], want, rtol=1e-6)
    eng.close()
    sim.operations.integrator = integ
    sim.run(0)
    np.testing.assert_allclose(y.energies, want, rtol=1e-6)
    sim.close()
