"""One particle at infinity, at minus infinity and at NaN of either sign: its pairs are
outside every cutoff, so the FP64 forces and gradients of all other particles are those
without it (the oracle's comparisons reject the pair)."""

import ctypes

import numpy as np
import pytest

import azplugins_gb300 as az
from helpers import box_of, force_error, random_fluid
from test_gpu_walk64 import PAIRS, _forces, _setup

pytestmark = pytest.mark.gpu

BAD = {"inf": np.inf, "-inf": -np.inf, "nan": np.nan, "-nan": np.copysign(np.nan, -1.0)}


def _moved(x, value, axes):
    m = x.copy()
    m[len(x) // 2, axes] = value
    return m


@pytest.mark.parametrize("axes", [[0], [0, 1, 2]])
@pytest.mark.parametrize("bad", sorted(BAD))
@pytest.mark.parametrize("kind", sorted(PAIRS))
def test_pair_forces(orc, kind, bad, axes):
    x, typ, L, rec, rc = _setup(600, kind=kind)
    m = _moved(x, BAD[bad], axes)
    f, w = _forces(x, typ, L, rec, rc, kind, 4, moved=m)
    p4 = np.concatenate([m, typ[:, None].astype(float)], axis=1)
    box, nt = np.full(3, L), 2
    padded = np.zeros((2, 2, 4))
    padded[:, :, : rec.shape[2]] = rec
    start, idx = orc.nlist(p4, typ.astype(np.int32), nt, box, rc * rc, method="brute")
    F, U, W = orc.pair_forces(p4, typ.astype(np.int32), nt, box, start, idx, kind, padded, rc * rc, (0.8 * rc) ** 2,
                              "shift")
    # sums of at most 60 FP64 terms in another order
    for a, b in ((f[:, :3], F), (f[:, 3], U), (w.T, W)):
        assert np.isfinite(a).all()
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


@pytest.mark.parametrize("bad", sorted(BAD))
@pytest.mark.parametrize("kind", sorted(PAIRS))
@pytest.mark.parametrize("mode", [1, 2])
def test_gradients(kind, bad, mode):
    x, typ, L, rec, rc = _setup(500, kind=kind)
    grad = np.random.Generator(np.random.PCG64(2)).normal(size=(len(x), 4))
    k = len(x) // 2
    gx, gp = _forces(x, typ, L, rec, rc, kind, 4, moved=_moved(x, BAD[bad], [0, 1, 2]), mode=mode, grad=grad)
    rest = np.arange(len(x)) != k
    rx, rp = _forces(x[rest], typ[rest], L, rec, rc, kind, 4, mode=mode, grad=grad[rest])
    # the same terms, dealt to the lanes in another order
    for a, b in ((gx[rest], rx), (gp[rest], rp)):
        assert np.isfinite(a).all()
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


def _dpd_snapshot(N, seed):
    snap = random_fluid(N, 3.0, seed=seed, ntypes=2, min_dist=0.2)
    snap.particles.mass = np.ones(N)
    return snap


def _dpd_pot():
    pot = az.pair.DPDGeneralWeight(nlist=az.nlist.Cell(buffer=0.3), kT=1.5, default_r_cut=1.0)
    pot.params[("A", "A")] = dict(A=25.0, gamma=4.5, s=0.5)
    pot.params[("A", "B")] = dict(A=40.0, gamma=3.0, s=2.0)
    pot.params[("B", "B")] = dict(A=25.0, gamma=4.5, s=1.0)
    return pot


def _dpd_oracle(orc, snap, m, pot, ts, seed, dt):
    p = snap.particles
    rec, rc, _ = pot._tables(list(p.types))
    p4 = np.concatenate([m, np.asarray(p.typeid, dtype=float)[:, None]], axis=1)
    start, idx = orc.nlist(p4, p.typeid, 2, box_of(snap), rc * rc, method="brute")
    vel4 = np.concatenate([p.velocity, p.mass[:, None]], axis=1)
    return orc.dpd_forces(p4, vel4, p.typeid, np.arange(p.N, dtype=np.uint32), 2, box_of(snap), start, idx, rec, rc * rc,
                          1.5, dt, ts, seed)


@pytest.mark.parametrize("bad", sorted(BAD))
def test_dpd_driver(orc, bad):
    import torch

    from azplugins_gb300 import _compute, _lib

    snap, pot = _dpd_snapshot(700, 5), _dpd_pot()
    p = snap.particles
    rec, rc, _ = pot._tables(list(p.types))
    pos = _compute.device_positions(snap)
    vel = torch.ones((p.N, 4), dtype=torch.float64, device="cuda")
    vel[:, :3] = torch.from_numpy(p.velocity)
    tag = torch.arange(p.N, dtype=torch.int32, device="cuda")
    sysd = _compute.make_system(snap, pos, vel=vel.data_ptr(), tag=tag.data_ptr())
    nl = _compute.NeighborList(p.N, 2, rc, 0.3)
    nl.build(sysd)
    m = _moved(p.position, BAD[bad], [0, 1, 2])
    pos[:, :3] = torch.from_numpy(m)
    f = torch.zeros((p.N, 4), dtype=torch.float64, device="cuda")
    t = [torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda() for a in (rec, rc)]
    out = _lib.Forces()
    out.force, out.virial, out.virial_pitch, out.precision = f.data_ptr(), None, p.N, _lib.FP64
    _lib.check(_lib.load().azp_dpd_forces(ctypes.byref(sysd), nl.handle, t[0].data_ptr(), t[1].data_ptr(), 1.5, 0.01, 9, 4,
                                          ctypes.byref(out), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)),
               "azp_dpd_forces")
    F, U, W = _dpd_oracle(orc, snap, m, pot, 9, 4, 0.01)
    f = f.cpu().numpy()
    assert np.isfinite(f).all()
    assert force_error(f, F) < 1e-12
    nl.close()


@pytest.mark.parametrize("bad", sorted(BAD))
@pytest.mark.parametrize("system", ["dpd", "lj"])
def test_engine_forces(orc, system, bad):
    """A box of three cells a side, so that the particle is a list candidate of all."""
    from azplugins_gb300 import _engine

    if system == "dpd":
        snap, pot = _dpd_snapshot(230, 6), _dpd_pot()  # L 4.25
    else:
        snap = random_fluid(500, 0.6, seed=6, ntypes=2)  # L 9.41
        pot = az.pair.PerturbedLennardJones(nlist=az.nlist.Cell(buffer=0.4), default_r_cut=2.5, mode="shift")
        for a, b in (("A", "A"), ("A", "B"), ("B", "B")):
            pot.params[(a, b)] = dict(epsilon=1.0, sigma=1.0, attraction_scale_factor=0.5)
    p = snap.particles
    m = _moved(p.position, BAD[bad], [0, 1, 2])
    if system == "dpd":
        F, U, W = _dpd_oracle(orc, snap, m, pot, 9, 4, 0.005)
    else:
        rec, rc, ro = pot._tables(list(p.types))
        p4 = np.concatenate([m, np.asarray(p.typeid, dtype=float)[:, None]], axis=1)
        start, idx = orc.nlist(p4, p.typeid, 2, box_of(snap), rc * rc, method="brute")
        F, U, W = orc.pair_forces(p4, p.typeid, 2, box_of(snap), start, idx, "PerturbedLennardJones", rec, rc * rc, ro * ro,
                                  "shift")
    p.position = m
    p.acceleration = np.zeros((p.N, 3))
    sim = az.Simulation(seed=4, precision="fp64")
    sim.create_state_from_snapshot(snap)
    method = az.methods.LangevinFlow("all", kT=1.0, flow_field=az.flow.ConstantFlow((0.0, 0.0, 0.0)))
    integ = az.md.Integrator(dt=0.005, methods=[method], forces=[pot])
    eng = _engine.Engine(sim, integ, snap)
    eng.push(snap, 9)
    f = eng.forces()[0]
    assert np.isfinite(f).all()
    assert force_error(f, F) < 1e-12
    eng.close()
