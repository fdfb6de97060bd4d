"""The cluster kernel that steps small packings (rcpg_small.cu, N <= 8,192) at
the edges of its work split: one warp of particles, whole and ragged warps and
blocks, one to sixteen blocks, one to sixteen lanes per particle, the first
size that takes the step graph instead."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _packing(n, nd, ratio, walls, seed=5):
    import rcpgenerator_b200 as rb
    dist = {"type": "mono", "d": 1.0} if ratio == 1.0 else {"type": "bidisperse", "d1": 1.0, "d2": ratio, "p": 0.5}
    init = rb.initialize_particles({"phi": {2: 0.3, 3: 0.1, 4: 0.05}[nd], "N": n, "Ndim": nd, "box": [1.0] * nd,
                                    "walls": walls, "dist": dist, "seed": seed})
    return ({"positions": np.asarray(init["positions"]), "diameters": np.asarray(init["diameters"])},
            {"box": init["box"], "walls": init["walls"], "neighbor_max": 0})


CASES = [(1, 2, 1.0, [0, 0]), (31, 2, 1.4, [0, 0]), (33, 3, 1.0, [0, 0, 0]), (129, 2, 1.0, [1, 1]),
         (257, 3, 4.0, [-3, 0, 0]), (600, 4, 3.0, [0] * 4), (2049, 3, 1.0, [0, 0, 0]), (4100, 2, 1.4, [0, 0]),
         (8192, 3, 1.0, [0, 0, 0]), (8193, 3, 1.0, [0, 0, 0])]


@pytest.mark.parametrize("n,nd,ratio,walls", CASES)
def test_first_steps_track_the_exact_engine(cuda_device, n, nd, ratio, walls):
    """Two steps: the engines differ by the order of their sums, at most a few
    hundred ulps of the force on a particle whose contacts nearly cancel
    (1e-13), and a step moves a particle by half a smallest diameter at most."""
    import rcpgenerator_b200 as rb
    inp, cfg = _packing(n, nd, ratio, walls)
    a, b = (rb.run_packing_observed(inp, dict(cfg, engine=e), options={"max_steps": 2}, as_arrays=True)["result"]
            for e in ("exact", "graph"))
    assert a["steps"] == b["steps"] == 2
    assert np.array_equal(a["particle_origin"], b["particle_origin"])
    tol = 1e-12 * a["diameters"].min()
    assert np.abs(a["positions"] - b["positions"]).max() <= tol
    assert np.abs(a["diameters"] - b["diameters"]).max() <= tol


@pytest.mark.parametrize("n,nd,ratio,walls", [CASES[k] for k in (0, 1, 4, 6, 8)])
@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_slices_give_the_same_run(cuda_device, n, nd, ratio, walls, precision):
    """A run cut into launches of uneven length equals the uncut run bit for bit."""
    import rcpgenerator_b200 as rb
    inp, cfg = _packing(n, nd, ratio, walls)
    cfg["pair_precision"] = precision
    whole = rb.run_packing_observed(inp, cfg, options={"max_steps": 90}, as_arrays=True)["result"]
    eng = rb.PackingEngine(inp, cfg, {"max_steps": 90})
    for k in (1, 2, 31, 7, 0):
        eng.advance(k)
    cut = eng.result()
    eng.close()
    for key in ("positions", "diameters", "particle_origin", "phi_history", "force_history", "energy_history",
                "max_overlap_history"):
        assert np.array_equal(whole[key], cut[key], equal_nan=True), key
