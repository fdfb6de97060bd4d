"""overlap_report with box sides that give no minimum image (zero, infinite,
not a number) or a negative one, against the oracle, which restates the
reference's arithmetic: a quotient that is not a number drops the pair."""

from __future__ import annotations

import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
import overlap_oracle as oo  # noqa: E402

pytestmark = pytest.mark.gpu


class _State:
    def __init__(self, positions, diameters, box):
        self.positions, self.diameters, self.box = positions, diameters, box


# planar: every particle at the same coordinate along the last axis
@pytest.mark.parametrize("last", [0.0, np.inf, np.nan, -1.0, 1.0])
@pytest.mark.parametrize("planar", [True, False])
@pytest.mark.parametrize("nd", [2, 3])
def test_sides_without_a_minimum_image(cuda_device, nd, planar, last):
    from rcpgenerator_b200 import jobs
    rng = np.random.default_rng(11)
    n = 300
    pos = rng.random((n, nd))
    if planar:
        pos[:, -1] = 0.25
    D = rng.uniform(0.05, 0.12, n)
    box = np.array([1.0] * (nd - 1) + [last])
    P, S, M, nc = oo.overlap_pairs(pos, D, box)
    assert (nc > 0) == (abs(last) == 1.0)
    r = jobs.overlap_report(_State(pos, D, box))
    assert r["n_candidate_pairs"] == nc and r["n_overlapping"] == len(P)
    np.testing.assert_array_equal(np.asarray(r["pairs"]).reshape(-1, 2), P.reshape(-1, 2))
    np.testing.assert_array_equal(r["fractions_sum"], S)
    np.testing.assert_array_equal(r["fractions_min"], M)
