"""The arrays of a result: in the reference's order, independent of the engine
and of each other, and alive after both are gone."""

import gc

import numpy as np
import pytest

import rcpgenerator_b200 as rb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim,n", [(2, 33), (2, 255), (3, 257), (4, 1000), (3, 9001)])
def test_positions_outlive_engine_and_result(ndim, n):
    rng = np.random.default_rng(n)
    inp = {"positions": rng.random((n, ndim)), "diameters": rng.uniform(0.9, 1.1, n)}
    cfg = {"box": [1.0] * ndim, "walls": [0] * ndim}
    e = rb.PackingEngine(inp, cfg, {"max_steps": 4})
    e.advance(2)
    first, second = e.result(), e.result()
    kept = first["positions"].copy()
    assert first["positions"].shape == (n, ndim) and first["positions"].flags.writeable
    np.testing.assert_array_equal(first["positions"], second["positions"])
    second["positions"][:] = -1.0
    e.advance(2)
    assert not np.shares_memory(first["positions"], second["positions"])
    x = first["positions"]
    e.close()
    del first, second, e
    gc.collect()
    for _ in range(3):
        out = rb.run_packing_observed(inp, cfg, options={"max_steps": 2}, as_arrays=True)["result"]
    np.testing.assert_array_equal(x, kept)
    # particle_origin maps the result to the input: diameters keep their ratios
    ratio = out["diameters"] / inp["diameters"][out["particle_origin"].astype(np.int64)]
    np.testing.assert_allclose(ratio, ratio[0], rtol=1e-12)
