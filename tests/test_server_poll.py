"""Server.poll: a poll that finds no result allocates no result array; every result is an array of its own
(CPU, with a stand-in for the library)."""
import ctypes as C

import numpy as np

from cuda_multiddm_b200 import server as module
from cuda_multiddm_b200._lib import ChunkResult


class FakeLib:
    def __init__(self, results):
        self.results, self.pointers = list(results), []

    def ddm_server_poll(self, handle, sid, res, isf, capacity):
        self.pointers.append(isf)
        value = self.results.pop(0)
        if value is None:
            return 0
        C.memmove(isf, (C.c_double * capacity)(*[value] * capacity), 8 * capacity)
        return 1


def test_idle_polls_allocate_nothing_and_results_are_arrays_of_their_own(monkeypatch):
    fake = FakeLib([None, None, 1.0, None, 2.0, 3.0, 4.0])
    monkeypatch.setattr(module, "lib", lambda: fake)
    srv = module.Server.__new__(module.Server)
    srv._h, srv._isf, srv._res = None, {7: np.zeros(1000)}, ChunkResult()
    allocated = []
    for name in ("empty", "empty_like", "zeros", "zeros_like"):
        real = getattr(np, name)
        monkeypatch.setattr(np, name, lambda *a, real=real, **k: (allocated.append(1), real(*a, **k))[1])
    assert srv.poll(7) is None and srv.poll(7) is None and not allocated
    kept = [srv.poll(7)[1]]
    count = len(allocated)
    assert srv.poll(7) is None and len(allocated) == count
    kept.append(srv.poll(7)[1])
    view = srv.poll(7, copy=False)[1]
    assert view[0] == 3.0
    kept.append(srv.poll(7)[1])
    assert [k[0] for k in kept] == [1.0, 2.0, 4.0] and all((k == k[0]).all() for k in kept)
    assert not any(np.shares_memory(a, b) for i, a in enumerate(kept) for b in kept[:i])
