"""The fused step at every number of threads per particle against the oracle: rows
shorter and longer than a lane's queue, particle numbers off the block size, pairs
across the faces, two types, all modes, bonds."""

import os

import numpy as np
import pytest

import azplugins_gb300 as az
from helpers import box_of, force_error, oracle_system, pair_tables, random_fluid

pytestmark = pytest.mark.gpu

SIGMA = {("A", "A"): 1.0, ("A", "B"): 1.05, ("B", "B"): 1.1}


def _run(orc, N, rcut, mode, precision, tpp, bonds=False, steps=3):
    snap = random_fluid(N, 0.7, seed=N + 7, ntypes=2)
    p = snap.particles
    p.acceleration = np.zeros((N, 3))
    if bonds:
        L = box_of(snap)
        d = p.position[:-1:2] - p.position[1::2][: len(p.position[:-1:2])]
        d -= L * np.rint(d / L)
        near = np.nonzero((d * d).sum(axis=1) < 1.4 ** 2)[0]
        snap.resize_bonds(len(near))
        snap.bonds.types = ["b"]
        snap.bonds.group = np.stack([2 * near, 2 * near + 1], axis=1)
    lj = az.pair.PerturbedLennardJones(nlist=az.nlist.Cell(buffer=0.4), default_r_cut=rcut, default_r_on=0.8 * rcut,
                                       mode=mode)
    params = {k: dict(epsilon=1.0, sigma=s, attraction_scale_factor=0.5) for k, s in SIGMA.items()}
    for k, v in params.items():
        lj.params[k] = v
    forces = [lj]
    if bonds:
        dw = az.bond.DoubleWell()
        dw.params["b"] = dict(r_0=0.9, r_1=1.2, U_1=2.0, U_tilt=0.5)
        forces.append(dw)
    old = os.environ.get("AZP_TPP")
    if tpp:
        os.environ["AZP_TPP"] = str(tpp)
    try:
        sim = az.Simulation(seed=3, precision=precision)
        sim.create_state_from_snapshot(snap)
        m = az.methods.LangevinFlow("all", kT=1.0, flow_field=az.flow.ConstantFlow((0.1, 0.0, 0.0)))
        sim.operations.integrator = az.md.Integrator(dt=0.002, methods=[m], forces=forces)
        sim.run(steps)
    finally:
        if tpp:
            os.environ.pop("AZP_TPP")
            if old is not None:
                os.environ["AZP_TPP"] = old
    s = sim.state.get_snapshot()
    f, w = sim._engine.forces()
    rec, rc, ro = pair_tables(orc, "PerturbedLennardJones", params, ["A", "B"], {k: rcut for k in SIGMA},
                              {k: 0.8 * rcut for k in SIGMA})
    pair = dict(name="PerturbedLennardJones", params=rec, rcut=rc, ron=ro, mode=mode)
    bond = dict(name="DoubleWell", params=orc.bond_params("DoubleWell", dw.params["b"]).reshape(1, 8)) if bonds else None
    kw = dict(pair=pair, bond=bond, gamma=[1.0, 1.0], kT=1.0, dt=0.002, seed=3, flow_p=(0.1, 0.0, 0.0))
    md = orc.OracleMD(oracle_system(snap, p.acceleration), **kw)
    md.run(steps)
    dx = s.particles.position - md.s["pos4"][:, :3]
    dx -= box_of(snap) * np.rint(dx / box_of(snap))
    F, U, W = orc.OracleMD(oracle_system(s, s.particles.acceleration), **kw).forces()
    sim.close()
    return np.abs(dx).max(), force_error(f, F), abs(f[:, 3].sum() - U.sum()) / np.abs(U).sum(), np.abs(w - W).max() / np.abs(W).max()


@pytest.mark.parametrize("tpp", [0, 1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("N,rcut,mode", [(1025, 2.9, "shift"), (700, 1.2, "none"), (1501, 2.5, "xplor")])
def test_fp64_step_at_every_split(orc, N, rcut, mode, tpp):
    # FP64 sums of up to 130 terms in another order: 130 ulp of the largest term,
    # which exceeds the net force by less than a thousand times
    dx, f, u, w = _run(orc, N, rcut, mode, "fp64", tpp)
    assert dx < 1e-9 and f < 1e-10 and u < 1e-12 and w < 1e-11


@pytest.mark.parametrize("tpp", [1, 4, 32])
def test_fp64_step_with_bonds(orc, tpp):
    dx, f, u, w = _run(orc, 901, 1.5, "none", "fp64", tpp, bonds=True)
    assert dx < 1e-9 and f < 1e-10 and u < 1e-12 and w < 1e-11


@pytest.mark.parametrize("tpp", [0, 1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("N,rcut,mode", [(1025, 2.9, "shift"), (700, 1.2, "none"), (1501, 2.5, "xplor")])
def test_fp32_step_at_every_split(orc, N, rcut, mode, tpp):
    # the FP32 force budget of the other tests; the virial sums up to 130 FP32 terms
    dx, f, u, w = _run(orc, N, rcut, mode, "fp32", tpp)
    assert dx < 1e-6 and f < 1e-5 and u < 1e-6 and w < 1e-5


@pytest.mark.parametrize("tpp", [1, 4, 32])
def test_fp32_step_with_bonds(orc, tpp):
    dx, f, u, w = _run(orc, 901, 1.5, "none", "fp32", tpp, bonds=True)
    assert dx < 1e-6 and f < 1e-5 and u < 1e-6 and w < 1e-5
