"""The graph engine's row search (k_build_rows: rcpg_pairs_forces_scan where the
cell-unit search does not apply) against the sorted build (rcpg_pairs_full) on
the same state: the same partners for every particle, whatever the number of
lanes per particle, the size classes, grids narrower than a neighbourhood and
particles outside the box."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(n, nd, ratio, phi, stray, seed=7):
    rng = np.random.default_rng(seed)
    x = rng.random((n, nd))
    D = rng.uniform(1.0, ratio, n) ** -1.0 if ratio > 1 else np.ones(n)
    unit = np.pi ** (nd / 2) / {2: 1.0, 3: 1.3293403881791370, 4: 2.0, 5: 3.3233509704478426}[nd]
    D *= (phi / (unit * (D / 2) ** nd).sum()) ** (1.0 / nd)
    if stray:  # a few coordinates on and beyond the faces
        x[:: max(1, n // 9), 0] = -0.03
        x[1:: max(1, n // 7), nd - 1] = 1.02
        x[2:: max(1, n // 5), 0] = 0.0
    return x, D


# n: one particle, around a warp, each rule of search_lanes (32, 4 and 1 lanes; 4-D: 16 and 8)
@pytest.mark.parametrize("n,nd,ratio,phi,stray", [
    (1, 2, 1.0, 0.1, False), (2, 3, 1.0, 0.3, False), (33, 2, 1.3, 0.5, False), (63, 3, 1.0, 0.3, True),
    (129, 4, 2.0, 0.15, False), (500, 2, 12.0, 0.5, False), (4095, 3, 1.4, 0.3, False),
    (4097, 3, 9.0, 0.3, True), (19999, 3, 1.2, 0.33, False), (25001, 3, 10.0, 0.33, False),
    (32769, 3, 10.0, 0.33, True), (70001, 2, 8.0, 0.5, False), (5000, 4, 6.0, 0.15, True),
    (20001, 4, 5.0, 0.2, False), (1500, 5, 3.0, 0.05, False),
])
def test_row_search_finds_the_sorted_builds_partners(cuda_device, native, n, nd, ratio, phi, stray):
    import torch

    from tests import gpu_util as G
    x, D = _state(n, nd, ratio, phi, stray)
    box, walls = np.ones(nd), np.zeros(nd, np.int8)
    t = native.lib.rcpg_t_shell(G.hp(D), n)
    nbr, cnt, cap = G.pairs_full(x, D, box, walls, t, cap=64)
    want = G.rows_from(nbr, cnt, cap)
    xd, Dd = G.dev(x), G.dev(D)
    nbr2 = torch.zeros(cap * n, dtype=torch.int32, device="cuda:0")
    cnt2 = torch.zeros(n, dtype=torch.int32, device="cuda:0")
    F = torch.zeros(n * nd, dtype=torch.float64, device="cuda:0")
    need, fused = C.c_uint32(), C.c_int32()
    err = native.errbuf()
    rc = native.lib.rcpg_pairs_forces_scan(n, nd, G.vp(xd), G.vp(Dd), G.hp(box), G.hp(walls, G._i8p), t, 2.5e-4, 0,
                                           cap, G.vp(nbr2), G.vp(cnt2), C.byref(need), G.vp(F), G.hp(np.zeros(7)),
                                           C.byref(fused), None, err, len(err))
    native.raise_for(rc, err)
    assert fused.value == 0  # the row search, not the cell units
    got = [tuple(sorted(r)) for r in G.rows_from(nbr2, cnt2, cap)]
    if ratio > 2.5:
        # a particle outside the box sits in a boundary cell that its position does not belong to, and meets the
        # partners that the grid brings it: with several size classes (the graph engine's grids, not the sorted
        # build's one grid) these are others, so only pairs inside the box are compared
        out = set(np.nonzero(((x < 0.0) | (x > 1.0)).any(axis=1))[0])
        got, want = ([tuple(j for j in r if j not in out) for i, r in enumerate(rows) if i not in out]
                     for rows in (got, want))
    assert got == want
