"""A run whose last step opens with the spatial reorder takes that step, in
every engine and in the persistent batch kernel."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [60, 9001])
def test_run_ends_after_the_reorder_step(cuda_device, n):
    import rcpgenerator_b200 as rb
    rng = np.random.default_rng(n)
    inp = {"positions": rng.random((n, 2)), "diameters": rng.choice([1.0, 1.4], n)}
    cfg = {"box": [1.0, 1.0], "walls": [0, 0]}
    opt = {"max_steps": 20, "reorder_interval": 10}
    runs = [rb.run_packing_observed(inp, dict(cfg, engine=e), options=opt, as_arrays=True)["result"]
            for e in ("exact", "graph")]
    runs += [rb.run_packing_batch([(inp, cfg)], opt, concurrency=c)[0] for c in (-1, 1)]
    for r in runs:
        assert r["steps"] == 20 and len(r["phi_history"]) == 20
        np.testing.assert_array_equal(r["particle_origin"], runs[0]["particle_origin"])
