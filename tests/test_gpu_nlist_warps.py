"""The list build a warp per chunk (crowded stencil rows) against the oracle's
brute-force sets: particle numbers around the chunk and block sizes, boxes of 2 to 7
cells, rows beyond the shared-memory part, growth from a small list, types of different
reach, excluded partners, pairs at the list radius to the last bit."""

import numpy as np
import pytest

from helpers import box_of, pos4_of, random_fluid

pytestmark = pytest.mark.gpu


def _check(orc, snap, rcut, r_buff, exclusions=None, max_neighbors=64):
    from azplugins_gb300 import _compute

    N, nt = snap.particles.N, len(snap.particles.types)
    ex = None if exclusions is None else _compute.exclusions_csr(N, exclusions)
    sysd = _compute.make_system(snap, _compute.device_positions(snap))
    pos = _compute.device_positions(snap)
    sysd.pos = pos.data_ptr()
    nl = _compute.NeighborList(N, nt, rcut, r_buff, ex, max_neighbors=max_neighbors)
    nl.build(sysd)
    s, i = nl.to_csr()
    nl.close()
    rl = np.where(rcut > 0, rcut + r_buff, 0.0) ** 2
    so, io = orc.nlist(pos4_of(snap), snap.particles.typeid, nt, box_of(snap), rl, exclusions, method="brute")
    np.testing.assert_array_equal(s, so)
    np.testing.assert_array_equal(i, io)


@pytest.mark.parametrize("N", [60, 333, 1000, 2049, 4097])
@pytest.mark.parametrize("cells", [2.05, 3.1, 5.2, 7.4])
def test_boxes_of_few_cells(orc, N, cells):
    snap = random_fluid(N, 0.8, seed=N, min_dist=0.7)
    L = box_of(snap)[0]
    _check(orc, snap, np.array([[0.9 * L / cells]]), 0.1 * L / cells)


@pytest.mark.parametrize("max_neighbors", [8, 300])
def test_long_rows(orc, max_neighbors):
    # about 330 neighbours a particle: beyond the 192 of the shared-memory rows
    snap = random_fluid(3000, 0.8, seed=31, ntypes=2, min_dist=0.7)
    ex = np.array([[k, k + 1] for k in range(0, 2999, 3)])
    _check(orc, snap, np.array([[4.2, 4.2], [4.2, 1.0]]), 0.4, ex, max_neighbors)


def test_many_particles_take_eight_a_warp(orc):
    snap = random_fluid(40003, 0.9, seed=33, ntypes=2, min_dist=0.6)
    _check(orc, snap, np.array([[2.4, 2.0], [2.0, 1.1]]), 0.3, np.array([[k, k + 5] for k in range(0, 39000, 7)]))


def test_reach_by_type_and_types_never_listed(orc):
    snap = random_fluid(9000, 0.6, seed=34, ntypes=3, min_dist=0.6)
    _check(orc, snap, np.array([[0.9, 0.0, 2.5], [0.0, 0.0, 0.0], [2.5, 0.0, 5.0]]), 0.3)


def test_pairs_at_the_list_radius(orc):
    import azplugins_gb300 as az

    rng = np.random.Generator(np.random.PCG64(4))
    N, L, r = 6000, 13.0, 2.3
    base = rng.uniform(-0.5, 0.5, size=(N // 2, 3)) * L
    d = rng.normal(size=(N // 2, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    pos = np.concatenate([base, base + d * r * (1.0 + rng.uniform(-4e-16, 4e-16, size=(N // 2, 1)))])
    pos -= L * np.floor((pos + 0.5 * L) / L)
    snap = az.Snapshot(N)
    snap.particles.position = pos
    snap.configuration.box = [L, L, L, 0, 0, 0]
    _check(orc, snap, np.array([[2.0]]), 0.3)
