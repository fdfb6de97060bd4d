"""Runs whose rows outgrow their capacity on the way: advance(k) takes k steps,
every observation arrives, and the cut run equals the whole one, by the
cluster kernel (N <= 8,192) and by the step graph."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _input(n):
    rng = np.random.default_rng(9)
    D = np.ones(n)
    D[:: 450] = 20.0  # as dense as the small ones become, their neighbours line up around them
    return {"positions": rng.random((n, 2)), "diameters": D}, {"box": [1.0, 1.0], "walls": [0, 0]}


@pytest.mark.parametrize("n", [400, 9001])
def test_steps_and_observations_across_row_growth(cuda_device, n):
    import rcpgenerator_b200 as rb
    inp, cfg = _input(n)
    opt = {"max_steps": 4100, "initial_phi_target": 0.05}
    eng = rb.PackingEngine(inp, cfg, opt)
    capacity, steps = [eng.result()["engine_stats"]["row_capacity"]], 0
    for k in (1, 50, 32, 7, 64, 100, 31, 90, 25, 600, 333, 601, 66, 100, 2000):
        done = eng.advance(k)
        steps += k
        assert eng.steps == steps and done == (steps == 4100)
        capacity.append(eng.result()["engine_stats"]["row_capacity"])
    cut = eng.result()
    eng.close()
    assert capacity[-1] > capacity[0], (capacity, cut['phi'])  # the rows did grow
    seen = []
    out = rb.run_packing_observed(inp, cfg, progress_interval=25, callback=lambda u: seen.append(u["step"]),
                                  options=opt, as_arrays=True)["result"]
    assert seen == list(range(0, 4101, 25))
    for key in ("positions", "diameters", "particle_origin", "phi_history", "force_history"):
        assert np.array_equal(out[key], cut[key], equal_nan=True), key
