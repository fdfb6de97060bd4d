"""WarmStart.predict with a network that scales on the GPU: the rows it is
handed are those that the scaling on the host worked on."""

from __future__ import annotations

import numpy as np
import pytest

from rcpgenerator_b200 import warmstart as W


class _Scaling:
    """Stands in for the device network: both ways of scaling, on the host."""
    widths = (3, 4, 3)

    def forward(self, Xn):
        return np.asarray(Xn, dtype=np.float32)

    def predict(self, X, lo, hi, mean, std, y_mean, y_std):
        B, width = X.shape
        assert width == 3
        return self.forward((np.clip(X, lo, hi) - mean) / std).astype(np.float64) * y_std + y_mean


class _Forward:
    widths = _Scaling.widths
    forward = _Scaling.forward


# a list of rows, one row, one descriptor for every input, one per row
@pytest.mark.parametrize("X", [[[0.5, -3.0, 9.0], [2.0, 0.25, 3.0]], [0.5, -3.0, 9.0], 0.75, [[0.5], [2.0]]])
@pytest.mark.parametrize("held", [True, False])
def test_rows_of_every_accepted_shape(X, held):
    kw = dict(x_lo=np.array([0.0, -1.0, 2.0]), x_hi=np.array([1.0, 1.0, 5.0])) if held else {}
    a, b = (W.WarmStart(net, np.array([0.1, 0.2, 0.3]), np.array([1.0, 2.0, 4.0]), np.zeros(3), np.ones(3), **kw)
            for net in (_Scaling(), _Forward()))
    np.testing.assert_array_equal(a.predict(X), b.predict(X))


def test_rows_of_another_width_are_refused():
    ws = W.WarmStart(_Scaling(), np.zeros(3), np.ones(3), np.zeros(3), np.ones(3))
    with pytest.raises(ValueError):
        ws.predict([[1.0, 2.0]])
