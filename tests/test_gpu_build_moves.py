"""The two ways in which a graph-mode build brings the particles into cell order
(k_build_move: gathers after a per-cell sort, from 200,000 particles on, and
scattered moves below): the same run either way, and at the size of the first
gathers the rows of the sorted build."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("positions", "diameters", "particle_origin", "phi_history", "force_history", "energy_history",
        "max_overlap_history")


def _packing(n, nd, ratio, crowded):
    rng = np.random.default_rng(n)
    D = rng.uniform(1.0, ratio, n) if ratio > 1 else np.ones(n)
    x = rng.random((n, nd))
    if crowded:  # cells of far more than eight members, in every order of arrival
        x[: n // 8] = 0.3 + 0.02 * x[: n // 8]
    return {"positions": x, "diameters": D}, {"box": [1.0] * nd, "walls": [0] * nd, "neighbor_max": 4000}


# small and odd sizes, one and several size classes, crowded cells, the cell units and the row search, the line itself
@pytest.mark.parametrize("n,nd,ratio,crowded,precision", [
    (257, 2, 1.4, True, "f64"), (1023, 3, 6.0, False, "f64"), (2049, 4, 1.0, False, "mixed"), (9001, 2, 8.0, True, "mixed"),
    (20011, 3, 1.4, True, "f64"), (33333, 2, 1.0, True, "mixed"), (199_999, 2, 1.4, False, "mixed"),
    (200_001, 3, 6.0, False, "f64"),
])
def test_both_ways_give_the_same_run(cuda_device, native, n, nd, ratio, crowded, precision):
    import rcpgenerator_b200 as rb
    inp, cfg = _packing(n, nd, ratio, crowded)
    cfg["pair_precision"] = precision
    runs = []
    for gather in (0, 1):
        eng = rb.PackingEngine(inp, cfg, {"max_steps": 70, "reorder_interval": 40, "initial_phi_target": 0.1})
        native.lib.rcpg_engine_step_graph(eng._h, 1)
        native.lib.rcpg_engine_gather_builds(eng._h, gather)
        eng.advance(35)  # a replay and single steps
        eng.advance(0)
        runs.append(eng.result())
        eng.close()
    a, b = runs
    assert a["steps"] == b["steps"] == 70 and a["engine_stats"]["pair_builds"] == b["engine_stats"]["pair_builds"] > 20
    for key in KEYS:
        assert np.array_equal(a[key], b[key], equal_nan=True), key


@pytest.mark.parametrize("n,nd,ratio", [(200_001, 2, 1.4), (200_003, 3, 8.0)])
def test_rows_of_gathered_builds_are_the_sorted_builds(cuda_device, native, n, nd, ratio):
    """At the size of the first gathers, by the cell units and by the row search."""
    import ctypes as C

    import torch

    from tests import gpu_util as G
    inp, _ = _packing(n, nd, ratio, False)
    x, D = inp["positions"], inp["diameters"] * (0.1 / n) ** (1.0 / nd)
    box, walls = np.ones(nd), np.zeros(nd, np.int8)
    t = native.lib.rcpg_t_shell(G.hp(D), n)
    nbr, cnt, cap = G.pairs_full(x, D, box, walls, t, cap=64)
    xd, Dd = G.dev(x), G.dev(D)
    nbr2, cnt2 = torch.zeros_like(nbr), torch.zeros_like(cnt)
    F = torch.zeros(n * nd, dtype=torch.float64, device="cuda:0")
    need, fused = C.c_uint32(), C.c_int32()
    err = native.errbuf()
    rc = native.lib.rcpg_pairs_forces_scan(n, nd, G.vp(xd), G.vp(Dd), G.hp(box), G.hp(walls, G._i8p), t, 2.5e-4, 0, cap,
                                           G.vp(nbr2), G.vp(cnt2), C.byref(need), G.vp(F), G.hp(np.zeros(7)),
                                           C.byref(fused), None, err, len(err))
    native.raise_for(rc, err)
    assert fused.value == (1 if ratio < 2.5 else 0)
    want = G.rows_from(nbr, cnt, cap)
    assert sum(map(len, want)) > n  # the rows hold something
    assert [tuple(sorted(r)) for r in G.rows_from(nbr2, cnt2, cap)] == want
