"""The engine's host code (rcpg_engine.cu) on a stand-in for the CUDA runtime
and the kernels (tests/hostfake): no GPU."""

from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent / "hostfake"


@pytest.fixture(scope="module")
def lib():
    subprocess.run(["make", "-s", "-C", str(HERE)], check=True)
    lib = C.CDLL(str(HERE / "libhostfake.so"))
    u64, vp = C.c_uint64, C.c_void_p
    lib.hf_overflow.argtypes = [u64, C.c_uint32]
    lib.hf_reorder_every.argtypes = lib.hf_build_every.argtypes = [u64]
    lib.hf_engines.argtypes = [vp, u64]
    lib.hf_counts.argtypes = [C.POINTER(u64)]
    lib.hf_engine.restype, lib.hf_engine.argtypes = vp, [u64, C.c_int, C.c_double, C.c_int, C.c_int, C.c_int, u64, C.c_int]
    lib.hf_free.argtypes = [vp]
    lib.hf_advance.argtypes = [vp, u64]
    lib.hf_steps.restype, lib.hf_steps.argtypes = u64, [vp]
    lib.hf_run.restype, lib.hf_run.argtypes = u64, [vp, u64, C.POINTER(u64), u64]
    lib.hf_result.argtypes = [vp, C.POINTER(C.c_double)]
    yield lib
    lib.hf_set_device(0)


def _engine(lib, small, graph_steps=32, max_steps=100, overflows=(), exact=0, mixed=0, device=0, n=50, ndim=2, wide=1.0):
    lib.hf_reset(small)
    lib.hf_set_device(device)
    for step, need in overflows:
        lib.hf_overflow(step, need)
    e = lib.hf_engine(n, ndim, wide, exact, mixed, graph_steps, max_steps, device)
    assert e
    return e


# overflows in the middle of a slice, at its first and its last step, twice in a step's slice, at the last step of
# the run; by the small-packing kernel and by the step graph (replays of 32 and single steps)
OVERFLOWS = [[], [(7, 40)], [(1, 40)], [(5, 40)], [(6, 40)], [(40, 30), (41, 50)], [(100, 40)], [(33, 40), (64, 50)]]


@pytest.mark.parametrize("small", [1, 0])
@pytest.mark.parametrize("overflows", OVERFLOWS)
def test_advance_takes_the_steps_it_is_asked_for(lib, small, overflows):
    e = _engine(lib, small, overflows=overflows)
    steps = 0
    for k in (5, 1, 1, 33, 2, 40, 7, 32):
        done = lib.hf_advance(e, k)
        steps = min(steps + k, 100)
        assert (lib.hf_steps(e), done) == (steps, int(steps == 100))
    lib.hf_free(e)


@pytest.mark.parametrize("small", [1, 0])
@pytest.mark.parametrize("overflows", OVERFLOWS)
def test_every_observation_of_a_run_arrives(lib, small, overflows):
    e = _engine(lib, small, overflows=overflows)
    out = (C.c_uint64 * 64)()
    n = lib.hf_run(e, 5, out, 64)
    assert list(out[:n]) == list(range(0, 101, 5))
    lib.hf_free(e)


@pytest.mark.parametrize("small", [1, 0])
@pytest.mark.parametrize("every", [100, 50, 20, 99])
def test_a_reorder_at_the_last_step_does_not_end_the_run_before_it(lib, small, every):
    e = _engine(lib, small)
    lib.hf_reorder_every(every)
    assert lib.hf_advance(e, 0) == 1 and lib.hf_steps(e) == 100
    lib.hf_free(e)


@pytest.mark.parametrize("exact,mixed,small", [(1, 0, 0), (0, 0, 0), (0, 0, 1), (0, 1, 0), (0, 1, 1)])
@pytest.mark.parametrize("device", [0, 1])
def test_work_goes_to_the_engines_device_whatever_is_current(lib, exact, mixed, small, device):
    """Steps, observations and results with the other device current: everything is launched and allocated on the
    engine's device, the pending ADAM pass of the exact engine among it, and the caller's device stays current."""
    e = _engine(lib, small, exact=exact, mixed=mixed, overflows=[(9, 40)], device=device)
    other = 1 - device
    lib.hf_set_device(other)
    passes = C.c_double()
    lib.hf_leave_error()  # by a call of the caller's own
    assert lib.hf_advance(e, 12) == 0 and lib.hf_get_device() == other
    assert lib.hf_result(e, C.byref(passes)) == 0 and lib.hf_get_device() == other
    if exact:
        assert passes.value == 0.5 + 12  # the stand-in ADAM pass adds one
    out = (C.c_uint64 * 64)()
    n = lib.hf_run(e, 5, out, 64)
    # step 0 is reported at the start of the call
    assert list(out[:n]) == [0] + list(range(15, 101, 5)) and lib.hf_get_device() == other
    assert lib.hf_observer_device() == other
    counts = (C.c_uint64 * 4)()
    lib.hf_counts(counts)
    assert counts[0] == 0
    lib.hf_free(e)


@pytest.fixture(scope="module")
def small():
    subprocess.run(["make", "-s", "-C", str(HERE), "libsmallfit.so"], check=True)
    lib = C.CDLL(str(HERE / "libsmallfit.so"))
    lib.sf_ok.argtypes = [C.c_uint64, C.c_int, C.c_uint32, C.c_int, C.c_int, C.c_int]
    return lib


@pytest.mark.parametrize("nd", range(2, 9))
def test_cluster_kernel_only_where_its_cluster_fits(small, nd):
    """A device without room for the cluster (or a refusal of its shared memory or size) leaves small packings to the
    step graph, without an error; larger packings and grids never ask."""
    for n, blocks in ((64, 1), (2000, 16), (8192, 16)):
        assert small.sf_ok(n, nd, 500, 1, 0, 0) == 1 and small.sf_cluster() == blocks
        assert small.sf_ok(n, nd, 500, 0, 0, 0) == 0
        assert small.sf_ok(n, nd, 500, 1, 1, 0) == 0  # cudaFuncSetAttribute refuses
        assert small.sf_ok(n, nd, 500, 1, 0, 1) == 0  # the query fails
    assert small.sf_ok(8193, nd, 500, 1, 0, 0) == 0 and small.sf_ok(8192, nd, 12288, 1, 0, 0) == 0
    assert small.sf_ok(8192, nd, 12287, 1, 0, 0) == 1


def test_cluster_kernel_reports_its_launch(small):
    assert small.sf_run(3, 0, 0) == 0
    assert small.sf_run(3, 1, 0) == 1 and small.sf_run(3, 0, 701) == 701 and small.sf_run(9, 0, 0) != 0


def test_engine_takes_the_step_graph_where_the_cluster_kernel_does_not_fit(lib):
    for fits in (0, 1):
        e = _engine(lib, fits)
        counts = (C.c_uint64 * 4)()
        assert lib.hf_advance(e, 0) == 1 and lib.hf_steps(e) == 100
        lib.hf_counts(counts)
        assert (counts[1] > 0, counts[3] > 0) == (not fits, bool(fits))
        lib.hf_free(e)


def test_graph_of_any_length_takes_few_launches(lib):
    """graph_steps steps between two looks, whatever divides them: no graph of fewer than four steps unless there are
    no more, no more launches than one per four steps, and no larger graph than the steps themselves."""
    for graph_steps in list(range(1, 70)) + [97, 128, 1009]:
        e = _engine(lib, 0, graph_steps=graph_steps, max_steps=2 * graph_steps)
        counts = (C.c_uint64 * 4)()
        assert lib.hf_advance(e, graph_steps) == (0 if graph_steps else 1) and lib.hf_steps(e) == graph_steps
        lib.hf_counts(counts)
        launches, captured = counts[1], counts[2]
        assert launches * captured == graph_steps
        assert captured >= min(4, graph_steps)
        assert captured <= max(8, min(d for d in range(4, graph_steps + 1) if graph_steps % d == 0)
                               if graph_steps >= 4 else 3)
        lib.hf_free(e)


# (ndim, width of the size distribution, engines at once): particles up to which the cluster kernel takes every step
@pytest.mark.parametrize("ndim,wide,engines,limit", [
    (2, 1.0, 1, 8192), (3, 9.0, 1, 8192), (4, 1.0, 1, 3500), (4, 9.0, 1, 1500), (4, 9.0, 8, 8192), (5, 1.0, 7, 1200),
    (5, 1.0, 32, 2500), (6, 9.0, 1, 1000), (6, 1.0, 32, 2500), (7, 1.0, 1, 1000), (8, 1.0, 1, 700), (8, 1.0, 32, 1200),
])
def test_path_of_small_packings(lib, ndim, wide, engines, limit):
    """Above the limit the share of rebuilding steps decides: at most 0.9 (limit / N)^2 of the last 64 or more. The first
    64 steps are the step graph's above 1.5 times the limit."""
    for n in (m for m in (limit - 1, limit, limit + 1, 2 * limit) if m <= 8192):  # more never ask for it
        for every in (1, 8, 2, 64):
            e = _engine(lib, 1, max_steps=384, n=n, ndim=ndim, wide=wide)
            lib.hf_engines(e, engines)
            lib.hf_build_every(every)
            assert lib.hf_advance(e, 0) == 1 and lib.hf_steps(e) == 384
            counts = (C.c_uint64 * 4)()
            lib.hf_counts(counts)
            steps_of_graph = counts[1] * counts[2]
            if n <= limit:
                assert (steps_of_graph, counts[3]) == (0, 1)
            elif n == limit + 1:  # by the cluster kernel at once
                assert (steps_of_graph, counts[3]) == ((320, 1) if every == 1 else (0, 6))
            else:  # by the step graph at once
                assert (steps_of_graph, counts[3]) == ((384, 0) if every <= 2 else (64, 5))
            lib.hf_free(e)
