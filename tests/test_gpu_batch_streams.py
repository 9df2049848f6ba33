"""A batch used from more than one place: its state read on another stream while a run is
under way, and its block size and lanes chosen beside a run and inside a capture."""

import ctypes

import numpy as np
import pytest

import azplugins_gb300 as az
from helpers import random_fluid

pytestmark = pytest.mark.gpu


def _batch(precision="fp32"):
    from azplugins_gb300.batch import ReplicaBatch

    snaps = []
    for k in range(6):
        s = random_fluid(1500 + 700 * k, 0.5, seed=k, min_dist=0.9)
        s.particles.acceleration = np.zeros((s.particles.N, 3))
        snaps.append(s)
    return ReplicaBatch(snaps, az.pair.ExpandedYukawa, [dict(epsilon=1.0, kappa=1.2, delta=0.1)] * 6, [1.3] * 6,
                        list(range(6)), dt=0.005, r_buff=0.2, precision=precision)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_reads_on_another_stream_leave_the_state_alone(precision):
    """What such a read returns may be of two moments; the run goes on as if it had not been."""
    import torch

    out = []
    for read in (False, True):
        b = _batch(precision)
        b.run(1)
        torch.cuda.synchronize()
        other = torch.cuda.Stream()
        b.run(400, check=False)
        while read:
            with torch.cuda.stream(other):
                b.get_arrays()
            if torch.cuda.current_stream().query():
                break
        torch.cuda.synchronize()
        b.run(2)
        assert b.builds > 5
        out.append([np.array(x) for x in b.get_arrays()])
        b.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


def test_choices_allocate_nothing_and_wait_for_nothing():
    """Inside a capture of this thread, where allocations, copies and waits are errors."""
    import torch

    b, ref = _batch(), _batch()
    b.run(1)  # (too short for graphs, whose destruction a capture does not allow either)
    ref.run(1)
    torch.cuda.synchronize()
    x = torch.zeros(1000, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x.add_(1.0)
        b.set_block(128)
        b.set_tpp(8)
        b.set_block(64)
    g.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 1000.0
    # and beside a run that is under way
    b.run(200, check=False)
    b.set_block(512)
    b.run(50, check=False)
    b.set_block(128)
    b.run(50)
    for n in (200, 50, 50):
        ref.run(n)
    # the block size changes no particle's arithmetic
    for a, c in zip(b.get_arrays(), ref.get_arrays()):
        assert np.array_equal(a, c)
    b.close()
    ref.close()
