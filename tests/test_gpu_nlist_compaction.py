"""The compaction of the list build a warp per chunk, in every row: lattices whose shells
lie at the list radius to the last bits (candidates of the band around it) and excluded
partners, in rows inside and beyond the shared-memory part, against brute force."""

import numpy as np
import pytest

from helpers import box_of, pos4_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,shell,exclude", [(11, 6.0, False), (16, 5.0, True), (17, 9.0, True), (13, 17.0, True)])
def test_shells_at_the_list_radius_and_exclusions(orc, side, shell, exclude):
    import azplugins_gb300 as az
    from azplugins_gb300 import _compute

    N, L = side ** 3, float(side)
    g = np.arange(side) - 0.5 * L
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
    rng = np.random.Generator(np.random.PCG64(side))
    x = x[rng.permutation(N)]
    snap = az.Snapshot(N)
    # displacements of a few units in the last place: pairs of the shell on both sides
    snap.particles.position = x + rng.integers(-3, 4, size=x.shape) * np.spacing(np.abs(x))
    snap.configuration.box = [L, L, L, 0, 0, 0]
    pairs = np.array([[k, (k + d) % N] for k in range(0, N, 2) for d in (1, 7, 61)]) if exclude else None
    ex = None if pairs is None else _compute.exclusions_csr(N, pairs)
    rl = np.sqrt(shell)
    pos = _compute.device_positions(snap)
    nl = _compute.NeighborList(N, 1, np.array([[rl - 0.25]]), 0.25, ex, max_neighbors=64)
    so, io = orc.nlist(pos4_of(snap), snap.particles.typeid, 1, box_of(snap), np.array([[(rl - 0.25 + 0.25) ** 2]]), pairs,
                       method="brute")
    for _ in range(5):
        nl.build(_compute.make_system(snap, pos))
        s, i = nl.to_csr()
        np.testing.assert_array_equal(s, so)
        np.testing.assert_array_equal(i, io)
    nl.close()
