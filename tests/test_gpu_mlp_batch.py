"""Batches above 2^21 rows through the warm-start network's entry points: the
rows at the end are those of a small batch, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

B = (1 << 21) + 33  # 65,538 tiles of 32 rows


def test_batches_above_two_million_rows(cuda_device):
    from rcpgenerator_b200.warmstart import Network
    net = Network(widths=(3, 8, 2), seed=1)
    rng = np.random.default_rng(2)
    X = np.zeros((B, 3), np.float32)
    T = np.zeros((B, 2), np.float32)
    X[-64:], T[-64:] = rng.normal(size=(64, 3)), rng.normal(size=(64, 2))
    Y = net.forward(X)
    np.testing.assert_array_equal(Y[-64:], net.forward(X[-64:]))
    one, inf = np.ones(3), np.full(3, np.inf)
    P = net.predict(X.astype(np.float64), -inf, inf, 0 * one, one, np.zeros(2), np.ones(2))
    np.testing.assert_array_equal(P, Y.astype(np.float64))
    loss = float(net.train_step(X, T, lr=0.0, update=False))
    # FP32 terms (a few roundings each) and a tree of FP32 sums over 2^22 of them: below 30 * 2^-24
    np.testing.assert_allclose(loss, np.mean((Y.astype(np.float64) - T) ** 2), rtol=2e-6)
    grad = net.grad.cpu().numpy()
    # the other rows are at their targets: the gradient is that of the 64 rows as a batch of their own, times 64 / B,
    # up to the BF16 roundings of dz (2^-9 each, two layers, on either side)
    small = Network(widths=(3, 8, 2), seed=1)
    small.train_step(X[-64:], T[-64:], lr=0.0, update=False)
    want = small.grad.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(grad * (B / 64.0) - want) <= 2.0 ** -7 * np.linalg.norm(want)
