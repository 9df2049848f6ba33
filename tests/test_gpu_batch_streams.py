"""A batch used from more than one place: its state read on another stream while a run is
under way."""

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
