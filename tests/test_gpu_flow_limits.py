"""Parabolic flow between plates so far apart, or so close, that the reciprocal of their
distance is no ordinary number: y / H is a division there."""

import numpy as np
import pytest

import azplugins_gb300 as az
from helpers import random_fluid

pytestmark = pytest.mark.gpu


def _states(flow, precision, method):
    snap = random_fluid(500, 0.6, seed=2)
    snap.particles.acceleration = np.zeros((500, 3))
    lj = az.pair.PerturbedLennardJones(nlist=az.nlist.Cell(buffer=0.4), default_r_cut=2.5)
    lj.params[("A", "A")] = dict(epsilon=1.0, sigma=1.0, attraction_scale_factor=0.5)
    cls = az.methods.LangevinFlow if method == "langevin" else az.methods.BrownianFlow
    sim = az.Simulation(seed=5, precision=precision)
    sim.create_state_from_snapshot(snap)
    sim.operations.integrator = az.md.Integrator(dt=0.001, methods=[cls("all", kT=1.0, flow_field=flow)], forces=[lj])
    sim.run(7)
    p = sim.state.get_snapshot().particles
    sim.close()
    return p.position, p.velocity


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("method", ["langevin", "brownian"])
@pytest.mark.parametrize("separation", [np.inf, 1e308])
def test_plates_at_infinity_are_a_constant_flow(separation, method, precision):
    got = _states(az.flow.ParabolicFlow(mean_velocity=0.5, separation=separation), precision, method)
    ref = _states(az.flow.ConstantFlow((0.75, 0.0, 0.0)), precision, method)
    for a, b in zip(got, ref):
        assert np.isfinite(a).all()
        assert np.array_equal(a, b)


def test_batch_with_plates_at_infinity():
    from azplugins_gb300.batch import ReplicaBatch

    out = []
    for flow in (az.flow.ParabolicFlow(mean_velocity=0.5, separation=np.inf), az.flow.ConstantFlow((0.75, 0.0, 0.0))):
        snap = random_fluid(300, 0.5, seed=3)
        snap.particles.acceleration = np.zeros((300, 3))
        b = ReplicaBatch([snap], az.pair.ExpandedYukawa, [dict(epsilon=1.0, kappa=1.5, delta=0.1)], [2.0], [4], dt=0.001,
                         precision="fp64", flow=flow)
        b.run(5)
        out.append(b.get_arrays())
        b.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
