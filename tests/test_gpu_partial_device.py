"""Engines on a stream that has part of the device's multiprocessors only (a green context):
a run that does not fit there as one cooperative launch is taken step by step."""

import ctypes

import numpy as np
import pytest

import azplugins_gb300 as az
from helpers import random_fluid

pytestmark = pytest.mark.gpu


def _partial_stream(sms):
    """A stream of a green context with about `sms` multiprocessors, or None without support."""
    import torch

    torch.zeros(1, device="cuda")
    cu = ctypes.CDLL("libcuda.so.1")
    if not hasattr(cu, "cuGreenCtxCreate"):
        return None
    dev = ctypes.c_int(0)
    # (resource descriptions are opaque here; the buffers are larger than they are)
    whole, part, rest = (ctypes.create_string_buffer(1024) for _ in range(3))
    groups, desc, ctx, stream = ctypes.c_uint(1), ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    calls = [lambda: cu.cuDeviceGet(ctypes.byref(dev), torch.cuda.current_device()),
             lambda: cu.cuDeviceGetDevResource(dev, whole, 1),
             lambda: cu.cuDevSmResourceSplitByCount(part, ctypes.byref(groups), whole, rest, 0, sms),
             lambda: cu.cuDevResourceGenerateDesc(ctypes.byref(desc), part, 1),
             lambda: cu.cuGreenCtxCreate(ctypes.byref(ctx), desc, dev, 1),
             lambda: cu.cuGreenCtxStreamCreate(ctypes.byref(stream), ctx, 1, 0)]
    return stream if all(c() == 0 for c in calls) else None


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_run_on_part_of_the_device(precision):
    import torch

    from azplugins_gb300 import _engine, _lib

    stream = _partial_stream(16)
    if stream is None:
        pytest.skip("no green contexts here")
    out = []
    for s in (None, stream):
        snap = random_fluid(20000, 0.7, seed=2, min_dist=0.9)
        snap.particles.acceleration = np.zeros((20000, 3))
        sim = az.Simulation(seed=5, precision=precision)
        lj = az.pair.PerturbedLennardJones(nlist=az.nlist.Cell(buffer=0.4), default_r_cut=2.5)
        lj.params[("A", "A")] = dict(epsilon=1.0, sigma=1.0, attraction_scale_factor=0.5)
        m = az.methods.LangevinFlow("all", kT=1.0, flow_field=az.flow.ConstantFlow((0.0, 0.0, 0.0)))
        eng = _engine.Engine(sim, az.md.Integrator(dt=0.005, methods=[m], forces=[lj]), snap)
        eng.push(snap, 0)
        torch.cuda.synchronize()
        for _ in range(2):
            _lib.check(eng._L.azp_md_run(eng._md, 50, s), "azp_md_run")
        torch.cuda.synchronize()
        eng.pull(snap)
        out.append((snap.particles.position, snap.particles.velocity))
        eng.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
