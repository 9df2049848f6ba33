"""The persistent run (one cooperative launch for many timesteps) against the steps as a
graph replay: bitwise the same states, through list rebuilds with and without re-sorts,
runs of odd and even length, more steps than one launch takes, boxes of few and many
cells, crowded and sparse."""

import os

import numpy as np
import pytest

import azplugins_gb300 as az
from azplugins_gb300 import workloads
from helpers import random_fluid

pytestmark = pytest.mark.gpu


def _run(snap, forces, method, dt, precision, kernel, chunks, env=()):
    old = dict(os.environ)
    os.environ["AZP_RUN_KERNEL"] = "1" if kernel else "0"
    os.environ.update(env)
    try:
        sim = az.Simulation(seed=5, precision=precision)
        sim.create_state_from_snapshot(snap)
        sim.operations.integrator = az.md.Integrator(dt=dt, methods=[method], forces=forces)
        for c in chunks:
            sim.run(c)
    finally:
        os.environ.clear()
        os.environ.update(old)
    p = sim.state.get_snapshot().particles
    th = sim.thermo()
    sim.close()
    return p, th


def _compare(snap, forces, method, dt, precision, chunks, env=(), builds=2):
    snap.particles.acceleration = np.zeros((snap.particles.N, 3))
    a, ta = _run(snap, forces(), method(), dt, precision, True, chunks, env)
    b, tb = _run(snap, forces(), method(), dt, precision, False, chunks, env)
    for k in ("position", "velocity", "image", "acceleration"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    assert ta["nlist_builds"] == tb["nlist_builds"] and ta["nlist_builds"] >= builds
    assert ta["potential_energy"] == tb["potential_energy"]


def _lj(buffer, rcut, types=("A",), mode="none"):
    lj = az.pair.PerturbedLennardJones(nlist=az.nlist.Cell(buffer=buffer), default_r_cut=rcut, default_r_on=0.9 * rcut,
                                       mode=mode)
    for a in types:
        for b in types:
            lj.params[(a, b)] = dict(epsilon=1.0, sigma=1.0, attraction_scale_factor=0.5)
    return lj


def _langevin():
    return az.methods.LangevinFlow("all", kT=1.0, flow_field=az.flow.ConstantFlow((0.1, 0.0, 0.0)))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("N,buffer,rcut", [(343, 0.4, 2.5), (2049, 0.15, 1.2), (4097, 0.4, 3.0)])
def test_fluid(precision, N, buffer, rcut):
    snap = random_fluid(N, 0.7, seed=N, min_dist=0.9)
    _compare(snap, lambda: [_lj(buffer, rcut)], _langevin, 0.005, precision, [1, 2, 3, 37, 300])


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("every", ["1", "3"])
def test_melt_with_bonds_and_order_keeping_builds(precision, every):
    snap = workloads.lj_fluid(n_side=12, density=0.85, jitter=0.02, seed=4)
    n = snap.particles.N
    idx = np.arange(n).reshape(-1, 12)
    snap.resize_bonds(len(idx) * 11)
    snap.bonds.types = ["A-A"]
    snap.bonds.group = np.stack([idx[:, :-1].ravel(), idx[:, 1:].ravel()], axis=1)

    def forces():
        dw = az.bond.DoubleWell()
        dw.params["A-A"] = dict(r_0=0.95, r_1=1.2, U_1=2.0, U_tilt=0.5)
        return [_lj(0.2, 2.0 ** (1.0 / 6.0)), dw]

    _compare(snap, forces, _langevin, 0.005, precision, [5, 60], env={"AZP_SORT_EVERY": every}, builds=4)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_two_types_brownian_and_a_type_group(precision):
    snap = random_fluid(3000, 0.5, seed=8, ntypes=2, min_dist=0.9)
    snap.particles.diameter = np.where(snap.particles.typeid == 1, 2.0, 1.0)
    _compare(snap, lambda: [_lj(0.2, 2.0, ("A", "B"), "xplor")],
             lambda: az.methods.BrownianFlow(az.filter.Type(["A"]), kT=1.0, flow_field=az.flow.ConstantFlow((0.1, 0.0, 0.0)),
                                             alpha=3.0), 0.002, precision, [1, 30, 61])




@pytest.mark.parametrize("precision,N", [("fp64", 77824), ("fp64", 77825), ("fp32", 116736), ("fp32", 116737)])
def test_at_the_largest_size(precision, N):
    snap = random_fluid(N, 0.7, seed=1, min_dist=0.9)
    _compare(snap, lambda: [_lj(0.2, 1.2)], _langevin, 0.005, precision, [1, 23], builds=2)
