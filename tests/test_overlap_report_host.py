"""What overlap_report asks of memory and of the GPU call, on a stand-in for the
library: bounded room before the pairs are known, and their exact number after."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest


class _Lib:
    def __init__(self, pairs):
        self.pairs, self.capacities = pairs, []

    def rcpg_overlap_report(self, n, ndim, pos, D, box, ncand, nov, capacity, *rest):
        from rcpgenerator_b200 import _native as N
        self.capacities.append(capacity)
        C.cast(ncand, C.POINTER(C.c_uint64))[0] = self.pairs
        C.cast(nov, C.POINTER(C.c_uint64))[0] = self.pairs
        return N.RCPG_ENOSPC if self.pairs > capacity else 0


class _State:
    def __init__(self, n, ndim):
        self.positions, self.diameters, self.box = np.zeros((n, ndim)), np.ones(n), np.ones(ndim)


# a call for ordinary states; a second one beyond 2 ndim n pairs; large states count first
@pytest.mark.parametrize("n,ndim,pairs,capacities", [
    (1000, 3, 2500, [6000]), (1000, 3, 0, [6000]), (1000, 3, 7000, [6000, 7000]), (1_000_000, 3, 100, [6_000_000]),
    (2_000_000, 3, 100, [0, 100]), (3_000_000, 2, 500, [0, 500]), (1_100_000, 8, 0, [0]),
])
def test_room_for_the_pairs(monkeypatch, n, ndim, pairs, capacities):
    from rcpgenerator_b200 import _native as N
    from rcpgenerator_b200 import jobs
    lib = _Lib(pairs)
    monkeypatch.setattr(N, "lib", lib)
    r = jobs.overlap_report(_State(n, ndim))
    assert lib.capacities == capacities and r["n_overlapping"] == pairs
    assert all(24 * c <= max(24 * pairs, 24 << 23) for c in lib.capacities)
