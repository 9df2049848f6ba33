"""Rows that outgrow the list within a run nobody checks: a gas that condenses, with excluded
partners (rows are compacted past their capacity). The step reads the entries written and no
others, the error word says overflow, and the checked run grows the list and goes on."""

import os

import numpy as np
import pytest

import azplugins_gb300 as az
from helpers import random_fluid

pytestmark = pytest.mark.gpu


def _snapshot(n):
    s = random_fluid(n, 0.2, seed=7, min_dist=1.0)
    s.particles.acceleration = np.zeros((n, 3))
    s.particles.mass = np.ones(n)
    # a bond of no force excludes its pair; partners anywhere in the box
    s.resize_bonds(n // 2)
    s.bonds.types = ["A-A"]
    s.bonds.group = np.random.Generator(np.random.PCG64(1)).permutation(n)[: n // 2 * 2].reshape(-1, 2)
    return s


def _engine(snap, precision, rcut, kernel):
    from azplugins_gb300 import _engine as e

    sim = az.Simulation(seed=5, precision=precision)
    lj = az.pair.PerturbedLennardJones(nlist=az.nlist.Cell(buffer=0.4), default_r_cut=rcut)
    lj.params[("A", "A")] = dict(epsilon=12.0, sigma=1.0, attraction_scale_factor=1.0)
    dw = az.bond.DoubleWell()
    dw.params["A-A"] = dict(r_0=1.0, r_1=2.0, U_1=0.0, U_tilt=0.0)
    m = az.methods.LangevinFlow("all", kT=0.3, flow_field=az.flow.ConstantFlow((0.0, 0.0, 0.0)), default_gamma=2.0)
    old = dict(os.environ)
    os.environ["AZP_RUN_KERNEL"] = kernel
    try:
        return e.Engine(sim, az.md.Integrator(dt=0.002, methods=[m], forces=[lj, dw]), snap)
    finally:
        os.environ.clear()
        os.environ.update(old)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,rcut,kernel", [(600, 3.0, "1"), (600, 3.0, "0"), (3000, 2.0, "1"), (3000, 2.0, "0")])
def test_condensing_gas(precision, n, rcut, kernel):
    from azplugins_gb300 import _lib

    snap = _snapshot(n)
    eng = _engine(snap, precision, rcut, kernel)
    eng.push(snap, 0)
    for _ in range(40):
        eng.run_async(400)
        if eng.error_word() & _lib.EBIT_NLIST_OVERFLOW:
            break
    assert eng.error_word() & _lib.EBIT_NLIST_OVERFLOW
    # more steps with short rows: wrong forces, but no fault
    eng.run_async(400)
    with pytest.raises(_lib.AzpError) as err:
        eng.thermo()
    assert err.value.status == -3
    # the checked run grows the list
    eng.push(snap, 0)
    for _ in range(40):
        eng.run(400)
    assert eng.error_word() == 0
    assert np.isfinite(eng.thermo()["potential_energy"])
    eng.close()
