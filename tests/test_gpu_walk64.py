"""The FP64 drivers' FP32 scan of the caller's positions (csrc/walk64.cuh): forces and
gradients must not depend on it. Positions outside the box, coordinates at zero, type
pairs that are off, boxes of other scales, every number of threads per particle."""

import ctypes

import numpy as np
import pytest

from helpers import random_fluid

pytestmark = pytest.mark.gpu

PAIRS = {"PerturbedLennardJones": lambda s: [1.0, s, 0.5], "ExpandedYukawa": lambda s: [1.0, 1.2 / s, 0.1 * s],
         "Hertz": lambda s: [3.0]}


def _setup(N, scale=1.0, off=False, kind="PerturbedLennardJones"):
    from azplugins_gb300 import _lib

    snap = random_fluid(N, 0.6, seed=N, ntypes=2)
    x = snap.particles.position.copy()
    x[:3] = [[0.0, 0.0, 0.0], [0.0, 1.0, 0.0], [1.0, 0.0, -0.0]]
    x *= scale
    L = snap.configuration.box[0] * scale
    rec = np.zeros((2, 2, _lib.record_doubles(_lib.RECORD_PAIR, _lib.PAIR_KINDS[kind])))
    vals = np.array(PAIRS[kind](scale))
    for a in range(2):
        for b in range(2):
            v = vals.copy()
            if off and a != b:
                v[0] = 0.0
            _lib.check(_lib.load().azp_pair_params_from_values(_lib.PAIR_KINDS[kind], v.ctypes.data, rec[a, b].ctypes.data), "")
    rc = np.array([[2.5, 2.0], [2.0, 1.5]]) * scale
    return x, snap.particles.typeid, L, rec, rc


def _forces(x, typ, L, rec, rc, kind, tpp, moved=None, mode=1, grad=None):
    import torch

    from azplugins_gb300 import _compute, _lib

    N = len(x)
    pos = torch.zeros((N, 4), dtype=torch.float64, device="cuda")
    pos[:, :3] = torch.from_numpy(x)
    pos.view(torch.int64)[:, 3] = torch.from_numpy(typ.astype(np.int64)).cuda()
    s = _lib.System()
    s.N, s.ntypes, s.pos = N, 2, pos.data_ptr()
    for d in range(3):
        s.box.L[d] = L
    nl = _compute.NeighborList(N, 2, rc, 0.16 * rc.max(), tpp=tpp)
    nl.build(s)
    if moved is not None:
        pos[:, :3] = torch.from_numpy(moved)
    t = [torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda() for a in (rec, rc, 0.8 * rc)]
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if grad is not None:
        g = torch.from_numpy(grad).cuda()
        gp = torch.zeros((N, 3), dtype=torch.float64, device="cuda")
        gr = torch.zeros((N, 4), dtype=torch.float64, device="cuda")
        _lib.check(_lib.load().azp_pair_adjoint(ctypes.byref(s), nl.handle, _lib.PAIR_KINDS[kind], t[0].data_ptr(),
                                                t[1].data_ptr(), t[2].data_ptr(), mode, g.data_ptr(), gp.data_ptr(),
                                                gr.data_ptr(), st), "adjoint")
        return gp.cpu().numpy(), gr.cpu().numpy()
    f = torch.zeros((N, 4), dtype=torch.float64, device="cuda")
    w = torch.zeros((6, N), dtype=torch.float64, device="cuda")
    out = _lib.Forces()
    out.force, out.virial, out.virial_pitch, out.precision = f.data_ptr(), w.data_ptr(), N, _lib.FP64
    _lib.check(_lib.load().azp_pair_forces(ctypes.byref(s), nl.handle, _lib.PAIR_KINDS[kind], t[0].data_ptr(),
                                           t[1].data_ptr(), t[2].data_ptr(), mode, ctypes.byref(out), st), "forces")
    return f.cpu().numpy(), w.cpu().numpy()


def _oracle(orc, x, typ, L, rec, rc, kind, mode):
    p4 = np.concatenate([x, typ[:, None].astype(float)], axis=1)
    box = np.full(3, L)
    padded = np.zeros((2, 2, 4))
    padded[:, :, : rec.shape[2]] = rec
    start, idx = orc.nlist(p4, typ.astype(np.int32), 2, box, rc * rc)
    return orc.pair_forces(p4, typ.astype(np.int32), 2, box, start, idx, kind, padded, rc * rc, (0.8 * rc) ** 2,
                           ["none", "shift", "xplor"][mode])


def _close(f, w, F, U, W, tol):
    assert np.abs(f[:, :3] - F).max() <= tol * np.abs(F).max()
    assert np.abs(f[:, 3] - U).max() <= tol * np.abs(U).max()
    assert np.abs(w.T - W).max() <= tol * np.abs(W).max()


@pytest.mark.parametrize("kind", sorted(PAIRS))
@pytest.mark.parametrize("tpp,mode", [(1, 0), (2, 1), (4, 2), (8, 1), (16, 0), (32, 2)])
def test_forces_at_every_split(orc, kind, tpp, mode):
    x, typ, L, rec, rc = _setup(1003, off=tpp == 8, kind=kind)
    f, w = _forces(x, typ, L, rec, rc, kind, tpp, mode=mode)
    # sums of at most 60 FP64 terms in another order
    _close(f, w, *_oracle(orc, x, typ, L, rec, rc, kind, mode), 1e-12)


@pytest.mark.parametrize("scale", [1e-14, 1e-9, 1e6, 1e13])
def test_other_scales(orc, scale):
    kind = "PerturbedLennardJones"
    x, typ, L, rec, rc = _setup(700, scale=scale)
    f, w = _forces(x, typ, L, rec, rc, kind, 4)
    _close(f, w, *_oracle(orc, x, typ, L, rec, rc, kind, 1), 1e-12)


@pytest.mark.parametrize("shift", [1.0, 2.0, 1000.0])
def test_positions_outside_the_box(orc, shift):
    kind = "PerturbedLennardJones"
    x, typ, L, rec, rc = _setup(900)
    rng = np.random.Generator(np.random.PCG64(3))
    moved = x + shift * L * rng.integers(-1, 2, size=x.shape)
    f, w = _forces(x, typ, L, rec, rc, kind, 4, moved=moved)
    # the moved coordinates are rounded at shift L: 2^-53 of it in r, times 14 in the
    # force, of terms up to 100 times the largest net force
    _close(f, w, *_oracle(orc, x, typ, L, rec, rc, kind, 1), max(1e-12, 1400.0 * 2.0 ** -53 * 4.0 * shift * L))


@pytest.mark.parametrize("tpp", [1, 4, 32])
def test_adjoint_of_one_type_pair_per_particle_pair(tpp):
    """Two types with the same record give the one-type sums, whose gradient is
    combined once per particle."""
    x, typ, L, rec, rc = _setup(800)
    rc = np.full((2, 2), 2.2)
    grad = np.random.Generator(np.random.PCG64(9)).normal(size=(len(x), 4))
    two = _forces(x, typ, L, rec, rc, "PerturbedLennardJones", tpp, grad=grad)
    moved = _forces(x, typ, L, rec, rc, "PerturbedLennardJones", tpp, grad=grad,
                    moved=x + 2.0 * L * np.sign(x[:, ::-1]))
    ref = _forces(x, typ, L, rec, rc, "PerturbedLennardJones", 2, grad=grad)
    for a, b in zip(two, ref):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
    for a, b in zip(moved, ref):
        assert np.abs(a - b).max() <= 1400.0 * 2.0 ** -53 * 8.0 * L * np.abs(b).max()
