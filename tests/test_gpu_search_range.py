"""The FP32 tests ahead of the graph engine's neighbour searches (k_cells and
k_build_rows, through rcpg_pairs_forces_scan) over the coordinates that the
FP64 predicate takes: particles whole box sides outside the box, and boxes
whose squared lengths leave the range of FP32."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_UNIT = {2: np.pi / 4, 3: np.pi / 6, 4: np.pi ** 2 / 32}


def _state(n, nd, ratio, phi, seed=7):
    rng = np.random.default_rng(seed)
    D = rng.uniform(1.0, ratio, n) ** -1.0 if ratio > 1 else np.ones(n)
    D *= (phi / (_UNIT[nd] * D ** nd).sum()) ** (1.0 / nd)
    return rng.random((n, nd)), D


def _scan(native, x, D, box, t, cap):
    """Rows of the graph engine's build and whether the cell units made them."""
    import torch

    from tests import gpu_util as G
    n, nd = x.shape
    xd, Dd = G.dev(x), G.dev(D)
    nbr = torch.zeros(cap * n, dtype=torch.int32, device="cuda:0")
    cnt = torch.zeros(n, dtype=torch.int32, device="cuda:0")
    F = torch.zeros(n * nd, dtype=torch.float64, device="cuda:0")
    need, fused = C.c_uint32(), C.c_int32()
    err = native.errbuf()
    rc = native.lib.rcpg_pairs_forces_scan(n, nd, G.vp(xd), G.vp(Dd), G.hp(box), G.hp(np.zeros(nd, np.int8), G._i8p), t,
                                           2.5e-4, 0, cap, G.vp(nbr), G.vp(cnt), C.byref(need), G.vp(F),
                                           G.hp(np.zeros(7)), C.byref(fused), None, err, len(err))
    native.raise_for(rc, err)
    return G.rows_from(nbr, cnt, cap), bool(fused.value)


# on either side of a whole number of sides below and above the box: within a
# cutoff of the particles that the cells of the faces bring together
OFFSETS = [-1.0, -2.0, -3.0, 2.0, 3.0, 1.0]


@pytest.mark.parametrize("n,nd", [(20011, 2), (20011, 3), (70001, 2)])
def test_cell_units_keep_partners_of_particles_whole_sides_outside(cuda_device, native, n, nd):
    from tests import gpu_util as G
    x, D = _state(n, nd, 1.3, 0.4 if nd == 2 else 0.3)
    t = native.lib.rcpg_t_shell(G.hp(D), n)
    rng = np.random.default_rng(1)
    out = rng.permutation(n)[:600]
    for k, i in enumerate(out):  # just outside the face that the particle's cell lies at
        off = OFFSETS[k % len(OFFSETS)]
        axis = k % nd
        x[i, axis] = off + rng.uniform(-1.0, 1.0) * D.max()
    box = np.ones(nd)
    nbr, cnt, cap = G.pairs_full(x, D, box, np.zeros(nd, np.int8), t, cap=64)
    want = G.rows_from(nbr, cnt, cap)
    got, cells = _scan(native, x, D, box, t, cap)
    assert cells
    assert sum(len(want[i]) for i in out) > 600  # they have partners
    assert [tuple(sorted(r)) for r in got] == want


# cell units (2-D, 3-D), and the row search by one lane per particle with size classes
@pytest.mark.parametrize("n,nd,ratio,cells", [(20011, 2, 1.3, True), (20011, 3, 1.3, True), (32771, 3, 10.0, False),
                                              (70001, 2, 8.0, False)])
@pytest.mark.parametrize("power", [-300, -70, -60, -50, 60, 120, 300])
def test_rows_do_not_depend_on_the_unit_of_length(cuda_device, native, n, nd, ratio, cells, power):
    """Lengths scaled by a power of two: every FP64 operation scales exactly, so the rows are the same."""
    from tests import gpu_util as G
    x, D = _state(n, nd, ratio, 0.4 if nd == 2 else 0.3)
    t = native.lib.rcpg_t_shell(G.hp(D), n)
    want, c0 = _scan(native, x, D, np.ones(nd), t, 192)
    s = 2.0 ** power
    got, c1 = _scan(native, x * s, D * s, np.full(nd, s), t * s, 192)
    assert c0 == c1 == cells
    assert got == want
