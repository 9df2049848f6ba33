"""The host arrays of ReplicaBatch.get_arrays: nobody is handed memory that somebody else
still refers to, from any thread; memory that nobody refers to is used again and bounded.
The device calls are stand-ins, so no GPU is needed."""

import collections
import gc
import sys
import threading

import numpy as np

import azplugins_gb300 as az
from azplugins_gb300 import batch


class _Library:
    def azp_batch_set_state(self, *args):
        return 0

    def azp_batch_get_state(self, *args):
        return 0

    def azp_batch_destroy(self, *args):
        pass


def _batch(monkeypatch, n=50):
    monkeypatch.setattr(batch, "_stream", lambda: None)
    b = batch.ReplicaBatch.__new__(batch.ReplicaBatch)
    b._L, b._b, b.timestep = _Library(), 1, 0
    b.off = np.array([0, n], dtype=np.int64)
    b._free = collections.deque(maxlen=2)
    s = az.Snapshot(n)
    s.configuration.box = [10.0] * 3 + [0.0] * 3
    b.set_state([s])
    return b


def _address(a):
    return a.__array_interface__["data"][0]


def test_threads_hold_arrays_of_their_own(monkeypatch):
    b = _batch(monkeypatch)
    shared = []

    def work(k):
        for _ in range(400):
            arrays = b.get_arrays()
            for x in arrays:
                x.fill(k)
            for _ in range(3):
                if not all((x == k).all() for x in arrays):
                    shared.append(k)
                    return
            del arrays

    old = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(old)
    assert not shared


def test_views_and_other_users_keep_the_memory(monkeypatch):
    import torch

    b = _batch(monkeypatch)
    held = [b.get_arrays()[0][3:9, 1:], b.get_arrays()[1].T, torch.from_numpy(b.get_arrays()[2])[1:],
            memoryview(b.get_arrays()[3])]
    gc.collect()
    others = [b.get_arrays() for _ in range(6)]
    taken = [(_address(x), x.nbytes) for s in others for x in s]
    for h in held:
        a = np.asarray(h)
        lo = _address(a)
        assert not any(lo < p + n and p < lo + a.nbytes for p, n in taken)


def test_memory_is_used_again_and_bounded(monkeypatch):
    b = _batch(monkeypatch)
    first = b.get_arrays()
    where = _address(first[0])
    first = None
    again = b.get_arrays()
    assert _address(again[0]) == where
    sets = [b.get_arrays() for _ in range(7)]
    del sets, again
    gc.collect()
    assert len(b._free) == 2
    b.close()
    assert len(b._free) == 0


def test_changes_of_an_array_object_stay_with_it(monkeypatch):
    b = _batch(monkeypatch)
    a = b.get_arrays()
    a[0].setflags(write=False)
    del a
    assert [x.shape for x in b.get_arrays()] == [(50, 4), (50, 4), (50, 3), (50, 3)]
    assert all(x.flags.writeable and x.flags.c_contiguous and x.flags.aligned for x in b.get_arrays())
