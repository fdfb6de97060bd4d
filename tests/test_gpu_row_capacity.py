"""The reference's capacity check on a row that is longer than its particle's
capacity, where several lanes search the row together (k_build_rows with 4
lanes per particle): the partners after the particle in the reference's order
decide, on either side of the capacity, as in the sorted build."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K, CAP = 53, 51  # partners of the particle under test; 3-D capacity 50 + neighbor_max of equal particles


def _input(before, n=5001):
    """A particle with K partners on a sphere around it, `before` of them before it in the input; the others of the
    n particles are far from it and from another."""
    rng = np.random.default_rng(3)
    D = 0.01
    k = np.arange(K) + 0.5
    z, a = 1.0 - 2.0 * k / K, np.pi * (1.0 + 5.0 ** 0.5) * k
    r = np.sqrt(1.0 - z * z)
    c = np.array([0.5, 0.5, 0.5])
    shell = c + 1.45 * D * np.stack([r * np.cos(a), r * np.sin(a), z], axis=1)  # the shell's cutoff is 1.5 D
    grid = np.stack(np.meshgrid(*[(np.arange(18) + 0.5) / 18] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    grid = grid[np.abs(grid - c).max(axis=1) > 4 * D]
    x = np.concatenate([shell[:before], [c], shell[before:], rng.permutation(grid)[:n - K - 1]])
    return {"positions": x, "diameters": np.full(len(x), D)}


@pytest.mark.parametrize("engine", ["graph", "exact"])
@pytest.mark.parametrize("before", [0, 1, 2, 3, 30, 53])
def test_half_row_on_either_side_of_the_capacity(cuda_device, engine, before):
    import rcpgenerator_b200 as rb
    cfg = {"box": [1.0] * 3, "walls": [0] * 3, "neighbor_max": 1, "engine": engine}
    opt = {"max_steps": 1, "fix_diameter": True, "reorder_interval": 0}
    if K - before > CAP:
        with pytest.raises(RuntimeError, match=rf"particle {before} exceeded its neighbor capacity \({CAP} slots\)"):
            rb.run_packing_observed(_input(before), cfg, options=opt)
    else:
        r = rb.run_packing_observed(_input(before), cfg, options=opt, as_arrays=True)["result"]
        assert r["steps"] == 1
