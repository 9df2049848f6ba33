"""Which path a run takes: the persistent kernel where it is claimed (one launch per 256
steps), the graph where it is refused, and the same states from both, for every pair and
bond form, walls, barriers and temperature tables that the persistent kernel takes; the
line of its largest size on this device; runs that fail."""

import ctypes
import os

import numpy as np
import pytest

import azplugins_gb300 as az
from azplugins_gb300 import workloads
from helpers import random_fluid

pytestmark = pytest.mark.gpu


def _environment(env):
    old = dict(os.environ)
    os.environ.update(env)
    return old


def _restore(old):
    os.environ.clear()
    os.environ.update(old)


def _run(snap, forces, method, dt, precision, kernel, steps):
    old = _environment({"AZP_RUN_KERNEL": "1" if kernel else "0"})
    try:
        sim = az.Simulation(seed=5, precision=precision)
        sim.create_state_from_snapshot(snap)
        sim.operations.integrator = az.md.Integrator(dt=dt, methods=[method], forces=forces)
        sim.run(steps)
    finally:
        _restore(old)
    launches = sim._engine.last_launches
    p = sim.state.get_snapshot().particles
    builds = sim.thermo()["nlist_builds"]
    sim.close()
    return p, builds, launches


def _lj(types=("A",), rcut=2.5, buffer=0.4):
    lj = az.pair.PerturbedLennardJones(nlist=az.nlist.Cell(buffer=buffer), default_r_cut=rcut)
    for a in types:
        for b in types:
            lj.params[(a, b)] = dict(epsilon=1.0, sigma=1.0, attraction_scale_factor=0.5)
    return lj


def _yukawa():
    y = az.pair.ExpandedYukawa(nlist=az.nlist.Cell(buffer=0.3), default_r_cut=2.5)
    y.params[("A", "A")] = dict(epsilon=1.0, kappa=1.5, delta=0.2)
    return y


def _hertz():
    h = az.pair.Hertz(nlist=az.nlist.Cell(buffer=0.3), default_r_cut=1.5)
    h.params[("A", "A")] = dict(epsilon=20.0)
    return h


def _colloid():
    c = az.pair.Colloid(nlist=az.nlist.Cell(buffer=0.4), mode="shift")
    for (a, b), (A, a1, a2, rc) in {("A", "A"): (144.0, 0.0, 0.0, 3.0), ("A", "B"): (100.0, 0.0, 2.5, 6.0),
                                    ("B", "B"): (40.0, 2.5, 2.5, 10.0)}.items():
        c.params[(a, b)] = dict(A=A, a_1=a1, a_2=a2, sigma=1.0)
        c.r_cut[(a, b)] = rc
    return c


def _fluid(n=2000, ntypes=1):
    s = random_fluid(n, 0.6, seed=n, ntypes=ntypes, min_dist=0.9)
    s.particles.acceleration = np.zeros((n, 3))
    return s


def _colloids():
    # a cubic lattice, one site in 30 a colloid of radius 2.5 (spacing 6.5 among all sites)
    n, a = 10, 6.5
    g = (np.arange(n) - 0.5 * (n - 1)) * a
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
    s = az.Snapshot(n ** 3)
    s.particles.types = ["A", "B"]
    s.particles.position = x
    s.particles.typeid = (np.arange(n ** 3) % 30 == 0).astype(np.int32)
    s.particles.diameter = np.where(s.particles.typeid == 1, 5.0, 1.0)
    s.particles.velocity = np.random.Generator(np.random.PCG64(1)).normal(size=x.shape)
    s.particles.acceleration = np.zeros(x.shape)
    s.configuration.box = [n * a] * 3 + [0.0] * 3
    return s


def _melt():
    s = workloads.lj_fluid(n_side=12, density=0.85, jitter=0.02, seed=4)
    n = s.particles.N
    idx = np.arange(n).reshape(-1, 12)
    s.resize_bonds(len(idx) * 11)
    s.bonds.types = ["A-A"]
    s.bonds.group = np.stack([idx[:, :-1].ravel(), idx[:, 1:].ravel()], axis=1)
    s.particles.acceleration = np.zeros((n, 3))
    return s


def _quartic():
    b = az.bond.Quartic()
    b.params["A-A"] = dict(k=1434.3, r_0=1.5, b_1=-0.7589, b_2=0.0, U_0=67.2234, sigma=1.0, epsilon=1.0, delta=0.0)
    return b


def _walls():
    # planes just outside the box (L 14.9), their force linear below 0.7
    w = az.wall.LJ93([az.wall.Plane(origin=(0, -8.0, 0), normal=(0, 1, 0)), az.wall.Plane(origin=(0, 8.0, 0), normal=(0, -1, 0))])
    w.params["A"] = dict(A=0.5, sigma=1.0, r_cut=3.0, r_extrap=0.7)
    return w


def _barrier():
    b = az.external.PlanarHarmonicBarrier(location=az.variant.Ramp(6.0, 5.0, 0, 200))
    b.params["A"] = dict(k=3.0, offset=0.1)
    return b


def _langevin(kT=1.0):
    return az.methods.LangevinFlow("all", kT=kT, flow_field=az.flow.ConstantFlow((0.1, 0.0, 0.0)))


CASES = {
    "lj": (_fluid, lambda: [_lj()], _langevin, 0.005, ("fp64", "fp32")),
    "yukawa": (_fluid, lambda: [_yukawa()], _langevin, 0.005, ("fp64", "fp32")),
    "hertz": (_fluid, lambda: [_hertz()], _langevin, 0.005, ("fp64", "fp32")),
    "colloid": (_colloids, lambda: [_colloid()], _langevin, 0.005, ("fp64", "fp32")),
    "quartic melt": (_melt, lambda: [_lj(rcut=2.0 ** (1.0 / 6.0)), _quartic()], _langevin, 0.002, ("fp64", "fp32")),
    "walls": (_fluid, lambda: [_lj(rcut=1.2), _walls()], _langevin, 0.001, ("fp64",)),
    "moving barrier": (_fluid, lambda: [_lj(), _barrier()], _langevin, 0.005, ("fp64", "fp32")),
    "temperature table": (_fluid, lambda: [_lj()], lambda: _langevin(az.variant.Ramp(1.0, 2.0, 0, 100)), 0.005,
                          ("fp64", "fp32")),
}


@pytest.mark.parametrize("name,precision", [(n, p) for n in sorted(CASES) for p in CASES[n][4]])
def test_both_paths_give_the_same_states(name, precision):
    system, forces, method, dt, _ = CASES[name]
    steps = 280
    a, ba, la = _run(system(), forces(), method(), dt, precision, True, steps)
    b, bb, lb = _run(system(), forces(), method(), dt, precision, False, steps)
    # step one, two launches of up to 256 steps, the closing step; three launches to two steps
    assert la == 4 and lb >= 3 * (steps - 1) // 2
    assert ba == bb
    for k in ("position", "velocity", "image", "acceleration"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k


@pytest.mark.parametrize("precision,per_sm", [("fp64", 2), ("fp32", 3)])
def test_the_line_of_the_largest_size(precision, per_sm):
    """FP64: a thread per particle resident, 2 blocks of 256 an SM; FP32: a step's blocks
    resident, 3 an SM (at one thread per particle, which rows of 8 entries take)."""
    import torch

    N = per_sm * 256 * torch.cuda.get_device_properties(0).multi_processor_count
    for n, persistent in ((N, True), (N + 1, False)):
        snap = random_fluid(n, 0.7, seed=1, min_dist=0.9)
        snap.particles.acceleration = np.zeros((n, 3))
        launches = _run(snap, [_lj(rcut=1.2, buffer=0.2)], _langevin(), 0.005, precision, True, 31)[2]
        assert (launches == 3) == persistent, (n, launches)


def _engine(snap, forces, precision, env):
    from azplugins_gb300 import _engine as e

    sim = az.Simulation(seed=5, precision=precision)
    integ = az.md.Integrator(dt=0.005, methods=[_langevin()], forces=forces)
    old = _environment(env)
    try:
        return e.Engine(sim, integ, snap)
    finally:
        _restore(old)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_run_that_fails_leaves_what_the_graph_leaves(precision):
    """Particles that ask for a list build in the very step in which others leave the range of
    numbers: no build follows, whichever warp of a block saw the failure."""
    import torch

    def go(kernel):
        snap = _fluid(3000)
        snap.particles.velocity[::2] *= 60.0  # 0.3 a step: past half the buffer in the first
        # pairs at one place, moving together: their forces are not numbers, from the first evaluation on
        for x in (snap.particles.position, snap.particles.velocity):
            x[251::256] = x[250::256][: len(x[251::256])]
        eng = _engine(snap, [_lj()], precision, {"AZP_RUN_KERNEL": kernel})
        eng.push(snap, 0)
        eng.run_async(40)
        eng.pull(snap)
        out = np.zeros(9)
        status = eng._L.azp_md_thermo(eng._md, out.ctypes.data, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        word = eng.error_word()
        eng.close()
        p = snap.particles
        return (status, word, out[8]), p.position, p.velocity, p.image

    first = go("0")
    assert first[0][:2] == (-7, 4)
    for _ in range(5):
        other = go("1")
        assert other[0] == first[0]
        for a, b in zip(first[1:], other[1:]):
            assert np.array_equal(a, b, equal_nan=True)
