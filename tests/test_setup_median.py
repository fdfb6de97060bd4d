"""The run set-up's median (rank N/2 of the diameters) against a full sort: sizes
around the one from which it brackets the rank, and values that defeat the bracket."""

import ctypes as C

import numpy as np
import pytest


def _values(kind, n, rng):
    if kind == "uniform":
        return rng.uniform(0.5, 1.5, n)
    if kind == "sorted":
        return np.sort(rng.lognormal(0.0, 0.5, n))
    if kind == "constant":
        return np.full(n, 0.75)
    if kind == "two":
        return np.where(rng.random(n) < 0.5, 1.0, 1.4)
    if kind == "few":  # the rank falls on a long run of equal values
        return rng.choice([0.5, 1.0, 1.0, 1.0, 2.0], n)
    d = np.full(n, 2.0)  # every sampled value is small, most others are large
    d[:: max(1, n // 4096)] = rng.uniform(0.5, 1.0, len(d[:: max(1, n // 4096)]))
    return d


@pytest.mark.parametrize("n", [1, 2, 65535, 65536, 70001, 200003])
@pytest.mark.parametrize("kind", ["uniform", "sorted", "constant", "two", "few", "sampled"])
def test_setup_median(hostemu, kind, n):
    lib = hostemu.lib
    lib.hostemu_setup_median.restype = C.c_double
    lib.hostemu_setup_median.argtypes = [C.c_uint64, C.POINTER(C.c_double)]
    d = np.ascontiguousarray(_values(kind, n, np.random.default_rng(n)))
    got = lib.hostemu_setup_median(n, d.ctypes.data_as(C.POINTER(C.c_double)))
    assert got == np.sort(d)[n // 2]
