"""The cluster kernel of small packings and the step graph on the same packing:
every step's state and history, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _packing(n, nd, ratio, walls, side):
    rng = np.random.default_rng(n + nd)
    D = rng.uniform(1.0, ratio, n) if ratio > 1 else np.ones(n)
    box = np.full(nd, side)
    x = rng.random((n, nd)) * box
    return {"positions": x, "diameters": D}, {"box": box.tolist(), "walls": walls}


# one warp, ragged warps, one to sixteen blocks and lanes; size classes, flat walls, a curved container, a stretched
# height, a wide box (few builds) and the largest packing
@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("n,nd,ratio,walls,side,kw", [
    (31, 2, 1.4, [0, 0], 1.0, {}), (65, 3, 1.0, [0] * 3, 1.0, {}), (600, 4, 1.0, [0] * 4, 1.0, {}),
    (700, 2, 8.0, [1, 1], 1.0, {}), (900, 3, 1.4, [-3, 0, 0], 1.0, {}), (1500, 2, 1.4, [0, 1], 1.0, {"fix_height": True}),
    (2000, 3, 1.0, [0] * 3, 1.0, {}), (2500, 3, 6.0, [0] * 3, 1.0, {}), (3000, 2, 1.4, [0, 0], 30.0, {}),
    (4097, 3, 1.4, [1, 0, 0], 20.0, {}), (8192, 2, 1.0, [0, 0], 1.0, {}), (300, 5, 1.2, [0] * 5, 1.0, {}),
])
def test_cluster_kernel_and_step_graph_give_the_same_run(cuda_device, native, n, nd, ratio, walls, side, kw, precision):
    import rcpgenerator_b200 as rb
    inp, cfg = _packing(n, nd, ratio, walls, side)
    cfg = dict(cfg, pair_precision=precision, mixed_switch=1e-5, **kw)
    opt = {"max_steps": 120, "reorder_interval": 50}
    runs = []
    for step_graph in (0, 1):
        eng = rb.PackingEngine(inp, cfg, opt)
        native.lib.rcpg_engine_step_graph(eng._h, step_graph)
        launches = eng.kernel_launches
        eng.advance(40)
        # 40 steps are one launch of the cluster kernel, several kernels each by the step graph
        assert (eng.kernel_launches - launches > 40) == bool(step_graph)
        eng.advance(0)
        runs.append(eng.result())
        eng.close()
    a, b = runs
    assert a["steps"] == b["steps"] == 120
    for key in ("positions", "diameters", "particle_origin", "phi_history", "force_history", "energy_history",
                "max_overlap_history", "mu_history", "alpha_history", "mu_flag_history"):
        assert np.array_equal(a[key], b[key], equal_nan=True), key


def test_a_run_may_change_between_the_paths(cuda_device, native):
    import rcpgenerator_b200 as rb
    inp, cfg = _packing(1200, 3, 1.4, [0] * 3, 1.0)
    cfg["pair_precision"] = "mixed"
    whole = rb.run_packing_observed(inp, cfg, options={"max_steps": 150}, as_arrays=True)["result"]
    eng = rb.PackingEngine(inp, cfg, {"max_steps": 150})
    for k, k_steps in enumerate((3, 40, 33, 5, 0)):
        native.lib.rcpg_engine_step_graph(eng._h, k % 2)
        eng.advance(k_steps)
    cut = eng.result()
    eng.close()
    for key in ("positions", "diameters", "phi_history", "force_history", "energy_history", "max_overlap_history"):
        assert np.array_equal(whole[key], cut[key], equal_nan=True), key


@pytest.mark.parametrize("n,nd,ratio,side", [(1300, 5, 1.2, 20.0), (3600, 4, 1.0, 20.0), (1600, 4, 3.0, 1.0), (1100, 6, 1.2, 20.0)])
def test_paths_chosen_by_the_share_of_builds_give_the_same_run(cuda_device, native, n, nd, ratio, side):
    """Sizes above the line from which few builds decide: by slices of either path, as one run of the step graph."""
    import rcpgenerator_b200 as rb
    inp, cfg = _packing(n, nd, ratio, [0] * nd, side)
    cfg["neighbor_max"] = 3000
    runs = []
    for step_graph in (0, 1):
        eng = rb.PackingEngine(inp, cfg, {"max_steps": 500})
        native.lib.rcpg_engine_step_graph(eng._h, step_graph)
        eng.advance(0)
        runs.append(eng.result())
        eng.close()
    a, b = runs
    for key in ("positions", "diameters", "phi_history", "force_history", "energy_history", "max_overlap_history"):
        assert np.array_equal(a[key], b[key], equal_nan=True), key
