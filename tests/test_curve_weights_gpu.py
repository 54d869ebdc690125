"""The gradient of a curve belongs to the polyline points that the loss is taken at: the Bezier weights
of the backward pass are those of the forward pass's parameters, float32(i / 31 in float64)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F = np.float32


def _weights(i):
    t = F(1.0) if i >= 31 else F(i * (1.0 / 31.0))
    u = F(1.0) - t
    return F(u * u), F(F(F(2.0) * u) * t), F(t * t)


def _from_one_value(weights, got):
    """Some float32 g has float32(w g) == got for every weight: g is near got / w."""
    near = F(got[1] / weights[1])
    g = [near]
    for to in (F(-np.inf), F(np.inf)):
        v = near
        for _ in range(4):
            v = np.nextafter(v, to)
            g.append(v)
    return any(all(F(w * v) == r for w, r in zip(weights, got)) for v in g)


@pytest.mark.parametrize("sample", [1, 8, 16, 17, 21, 25, 29, 30])
def test_bezier_weights_of_one_sample(sample):
    """A curve that runs along a row and turns back at one sample, left of a one-pixel tile: that sample is
    the pixel's nearest point, so each control point's gradient is its weight there times one number."""
    from weft_b200.candidates import Cand
    from weft_b200.refine import StackSet

    rng = np.random.default_rng(sample)
    patches, stacks = [], []
    for _ in range(24):
        # x(t) = p0 + 2 t (c - p0) + t^2 (p0 - 2 c + p1) turns where t (2 c - p0 - p1) = c - p0
        p0, c, y = -6.0 - rng.random(), -1.5 + 0.2 * rng.random(), 0.1 + 0.2 * rng.random()
        p1 = 2.0 * c - p0 - (c - p0) * 31.0 / sample
        stacks.append([Cand(3, (p0, y, c, y, p1, y, 3.0), tuple(rng.uniform(0.2, 0.8, 3)), None, 0.8)])
        patches.append(rng.random((1, 1, 3), dtype=np.float32))
    ss, params = StackSet.from_stacks(patches, stacks)
    got = ss.loss_backward(params, torch.ones(ss.n, device=params.device)).cpu().numpy()
    w = _weights(sample)
    assert np.all(got[:, 0] != 0.0)
    for row in got:
        assert _from_one_value(w, row[0:6:2]) and _from_one_value(w, row[1:6:2])
