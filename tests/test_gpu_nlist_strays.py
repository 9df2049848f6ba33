"""A particle far outside the box, or not finite, among others in the list builds a warp per
chunk: the cell it is put into is not the cell of its fixed-point words, and the rows of
the particles there must not suffer."""

import numpy as np
import pytest

import azplugins_gb300 as az
from helpers import box_of, pos4_of, random_fluid

pytestmark = pytest.mark.gpu

# positions in units of the box edge; one value per axis
STRAYS = {"nan": [np.nan] * 3, "inf": [np.inf] * 3, "-inf": [-np.inf, 0.1, 0.2], "far": [3.3, -2.9, 5.45],
          "far in z": [0.1, 0.2, -40.7]}


@pytest.mark.parametrize("stray", sorted(STRAYS))
@pytest.mark.parametrize("N,cells", [(1500, 5.2), (3000, 7.4), (41000, 9.3)])
def test_rows_beside_a_stray(orc, N, cells, stray):
    from azplugins_gb300 import _compute

    snap = random_fluid(N, 0.8, seed=N, min_dist=0.7)
    L = box_of(snap)[0]
    # the first particle heads the rows of its cell
    x = snap.particles.position.copy()
    x[0] = np.array(STRAYS[stray]) * L
    snap.particles.position = x
    rl = L / cells
    pos = _compute.device_positions(snap)
    nl = _compute.NeighborList(N, 1, np.array([[0.9 * rl]]), 0.1 * rl)
    nl.build(_compute.make_system(snap, pos))
    s, i = nl.to_csr()
    nl.close()
    # the oracle without the particle
    rest = pos4_of(snap)[1:]
    so, io = orc.nlist(rest, snap.particles.typeid[1:], 1, box_of(snap), np.array([[(0.9 * rl + 0.1 * rl) ** 2]]),
                       method="brute")
    keep = i[s[1]:]
    rows = np.repeat(np.arange(N), np.diff(s))[s[1]:]
    own = keep != 0
    np.testing.assert_array_equal(keep[own] - 1, io)
    np.testing.assert_array_equal(np.bincount(rows[own] - 1, minlength=N - 1), np.diff(so))


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
def test_batch_beside_a_stray(precision, tol):
    from azplugins_gb300.batch import ReplicaBatch

    def accelerations(snap):
        b = ReplicaBatch([snap], az.pair.ExpandedYukawa, [dict(epsilon=1.0, kappa=0.7, delta=0.3)], [1.9], [3], dt=0.001,
                         kT=0.0, gamma=0.0, precision=precision)
        b.run(1, check=False)
        acc = b.get_arrays()[2]
        b.close()
        return acc

    N = 1500
    snap = random_fluid(N, 0.7, seed=9, min_dist=0.8)  # L 12.9: 5 cells
    snap.particles.acceleration = np.zeros((N, 3))
    snap.particles.velocity = np.zeros((N, 3))
    snap.particles.mass = np.ones(N)
    rest = az.Snapshot(N - 1)
    rest.configuration.box = snap.configuration.box
    for k in ("position", "velocity", "mass", "acceleration"):
        setattr(rest.particles, k, getattr(snap.particles, k)[1:])
    x = snap.particles.position.copy()
    x[0] = np.nan
    snap.particles.position = x
    a, b = accelerations(snap)[1:], accelerations(rest)
    assert np.isfinite(a).all()
    # the same terms; in FP32 the compensated sums may meet them in another order
    assert np.abs(a - b).max() <= tol * np.abs(b).max()
