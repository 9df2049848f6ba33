"""The bounded wait of the persistent run's grid barrier, with a limit so short that it runs
out: an error status, no further steps, and a state that can be set again."""

import os

import numpy as np
import pytest

import azplugins_gb300 as az
from helpers import random_fluid

pytestmark = pytest.mark.gpu


def _engine(snap, precision, env):
    from azplugins_gb300 import _engine as e

    sim = az.Simulation(seed=5, precision=precision)
    lj = az.pair.PerturbedLennardJones(nlist=az.nlist.Cell(buffer=0.4), default_r_cut=2.5)
    lj.params[("A", "A")] = dict(epsilon=1.0, sigma=1.0, attraction_scale_factor=0.5)
    m = az.methods.LangevinFlow("all", kT=1.0, flow_field=az.flow.ConstantFlow((0.0, 0.0, 0.0)))
    old = dict(os.environ)
    os.environ.update(env)
    try:
        return e.Engine(sim, az.md.Integrator(dt=0.005, methods=[m], forces=[lj]), snap)
    finally:
        os.environ.clear()
        os.environ.update(old)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_wait_that_runs_out(precision):
    from azplugins_gb300 import _lib

    snap = random_fluid(4097, 0.7, seed=2, min_dist=0.9)
    snap.particles.acceleration = np.zeros((4097, 3))
    start = {k: getattr(snap.particles, k).copy() for k in ("position", "velocity", "acceleration", "image")}
    eng = _engine(snap, precision, {"AZP_RUN_POLLS": "1"})
    for _ in range(2):
        eng.push(snap, 0)
        with pytest.raises(_lib.AzpError) as err:
            eng.run(300)
        assert err.value.status == -6
        assert eng.error_word() & _lib.EBIT_TIMEOUT
        with pytest.raises(_lib.AzpError) as err:
            eng.thermo()
        assert err.value.status == -6
    # the state set after it is the one that an engine without such a run has
    eng.push(snap, 0)
    fresh = _engine(snap, precision, {})
    fresh.push(snap, 0)
    for a, b in zip(eng.forces(), fresh.forces()):
        assert np.array_equal(a, b)
    eng.pull(snap)
    assert np.abs(snap.particles.position - start["position"]).max() < 1e-12
    fresh.close()
    eng.close()
    # the device and an engine with the ordinary limit are as before
    out = []
    for env in ({}, {"AZP_RUN_KERNEL": "0"}):
        eng = _engine(snap, precision, env)
        for k in start:
            setattr(snap.particles, k, start[k].copy())
        eng.push(snap, 0)
        eng.run(60)
        eng.pull(snap)
        out.append((snap.particles.position, snap.particles.velocity))
        eng.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
