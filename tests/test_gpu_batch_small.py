"""Many small replicas of unequal size in one batch (several share a block of the fused
step): accelerations against all pairs in 64 bits, at every block size and both precisions;
choices of block and lanes between runs change nothing but the split."""

import numpy as np
import pytest

import azplugins_gb300 as az

pytestmark = pytest.mark.gpu
EPS, KAPPA, DELTA, RC = 1.0, 1.2, 0.1, 1.5


def _snaps(sizes, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for n in sizes:
        L = max((n / 0.3) ** (1.0 / 3.0), 4.1)
        m = int(np.ceil(round(n ** (1.0 / 3.0), 9)))
        g = (np.arange(m) + 0.5) * (L / m) - 0.5 * L
        x = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
        x = x[rng.permutation(len(x))[:n]] + rng.uniform(-0.1, 0.1, (n, 3)) * (L / m)
        s = az.Snapshot(n)
        s.particles.position = x - L * np.floor(x / L + 0.5)
        s.particles.velocity = np.zeros((n, 3))
        s.particles.acceleration = np.zeros((n, 3))
        s.configuration.box = [L] * 3 + [0.0] * 3
        out.append(s)
    return out


def _reference(s):
    x, L = s.particles.position, s.configuration.box[0]
    d = x[:, None, :] - x[None, :, :]
    d -= L * np.rint(d / L)
    r = np.sqrt((d * d).sum(axis=-1))
    on = (r < RC) & (r > 0.0)
    q = np.where(on, r, 1.0)
    u = EPS * np.exp(-KAPPA * (q - DELTA)) / (q - DELTA)
    f = np.where(on, u * (KAPPA + 1.0 / (q - DELTA)) / q, 0.0)
    return (f[:, :, None] * d).sum(axis=1)


def _batch(snaps, precision):
    from azplugins_gb300.batch import ReplicaBatch

    S = len(snaps)
    return ReplicaBatch(snaps, az.pair.ExpandedYukawa, [dict(epsilon=EPS, kappa=KAPPA, delta=DELTA)] * S, [RC] * S,
                        list(range(S)), dt=1e-9, kT=0.0, gamma=0.0, precision=precision)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
@pytest.mark.parametrize("block,tpp", [(64, 1), (128, 32), (256, 1), (256, 16), (512, 8)])
def test_accelerations(precision, tol, block, tpp):
    sizes = [1, 2, 7, 8, 9, 31, 32, 33, 5, 64, 65, 3, 17] * 12 + [400, 1, 1, 1]
    snaps = _snaps(sizes, 3)
    ref = np.concatenate([_reference(s) for s in snaps])
    b = _batch(snaps, precision)
    for k, t in ((block, tpp), (256, 4), (block, tpp)):
        b.set_block(k)
        b.set_tpp(t)
        b.run(1)  # particles at rest, and a timestep in which they stay where they are
        acc = b.get_arrays()[2]
        # sums of at most 40 terms (FP64); FP32 forces with compensated sums
        assert np.abs(acc - ref).max() <= tol * np.abs(ref).max()
    b.close()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
@pytest.mark.parametrize("block", [64, 256, 512])
def test_accelerations_of_many_alike(precision, tol, block):
    """Enough particles with rows of one length for a thread per particle."""
    snaps = _snaps([27, 33, 32, 1, 30] * 650, 4)
    ref = np.concatenate([_reference(s) for s in snaps])
    b = _batch(snaps, precision)
    b.set_block(block)
    b.run(1)
    acc = b.get_arrays()[2]
    assert np.abs(acc - ref).max() <= tol * np.abs(ref).max()
    if precision == "fp64":
        b.set_tpp(4)  # lanes on request
        b.run(1)
        assert np.abs(b.get_arrays()[2] - ref).max() <= tol * np.abs(ref).max()
    b.close()


def test_both_forms_of_the_fp32_step_agree_bitwise():
    """Without a list build on the way: a batch builds for all when one particle asks, so the
    larger one would sort its particles at other steps."""
    from azplugins_gb300.batch import ReplicaBatch

    snaps = _snaps([200, 216, 190, 225] * 110, 6)  # 91,410 particles
    out, builds = [], []
    for count in (440, 12):
        b = ReplicaBatch(snaps[:count], az.pair.ExpandedYukawa, [dict(epsilon=EPS, kappa=KAPPA, delta=DELTA)] * count,
                         [RC] * count, list(range(count)), dt=0.002, kT=1.0, r_buff=0.4, precision="fp32")
        b.run(30)
        builds.append(b.builds)
        out.append([np.array(x[: b.off[12]]) for x in b.get_arrays()])
        b.close()
    assert builds[0] == builds[1]
    for x, y in zip(*out):
        assert np.array_equal(x, y)


def test_autotune_in_fp32_times_a_block_size_once():
    b = _batch(_snaps([50, 60, 70], 5), "fp32")
    ran = []
    run = b.run
    b.run = lambda steps, check=True: (ran.append((b.block, b.tpp)), run(steps, check))
    res = b.autotune(candidates=(1, 2, 4), steps=3, repeats=1, blocks=(128, 256))
    assert set(res) == {(t, k) for t in (1, 2, 4) for k in (128, 256)}
    assert len(set(ran)) == 2 and len(ran) == 4
    del b.run
    b.close()
