"""Candidates that cannot win are left out of the scoring: the selections stay those of scoring every
candidate (the oracle's), whatever the pools hold, and the bound on a curve's error holds."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import fit as ofit
from oracle import render as orender


def _cand(rng, kind, s, wild):
    from weft_b200.candidates import Cand

    lo, hi = (-3.0, s + 3.0) if wild else (0.0, s - 1.0)
    n = {0: 0, 1: 4, 2: 4, 3: 6, 4: 6}[kind]
    g = [float(np.float32(v)) for v in rng.uniform(lo, hi, n)]
    if wild and n and rng.random() < 0.2:
        g = g[:2] * (n // 2)  # every point the same: a dot, a degenerate triangle
    g += {2: [float(rng.uniform(0.2, 3.0))], 3: [float(rng.uniform(0.2, 3.0))]}.get(kind, [])
    a, b = (-0.3, 1.4) if wild else (0.0, 1.0)
    c1 = tuple(float(np.float32(v)) for v in rng.uniform(a, b, 3)) if kind == 1 else None
    return Cand(kind, tuple(g), tuple(float(np.float32(v)) for v in rng.uniform(a, b, 3)), c1,
                float(np.float32(rng.uniform(a, b) if wild else rng.choice([1.0, 0.7, 0.4, 0.2]))))


def _workload(seed, sides, kinds, n, wild):
    rng = np.random.default_rng(seed)
    patches = []
    for s in sides:
        base = rng.random(3)
        edge = (np.arange(s)[:, None] + np.arange(s)[None, :] * rng.uniform(-1, 1) > s * rng.uniform(0.2, 0.8))[..., None]
        img = base + edge * rng.uniform(-0.5, 0.5, 3) + rng.normal(0.0, 0.02, (s, s, 3))
        patches.append(np.clip(img, 0.0, 1.0).astype(np.float32))
    pools = [[_cand(rng, int(k), s, wild) for k in rng.choice(kinds, n)] for s in sides]
    for p, pool in zip(patches, pools):  # colours that fit, so that candidates of every kind come close
        for c in pool[::2]:
            c.color0 = tuple(float(v) for v in p[int(rng.integers(p.shape[0])), int(rng.integers(p.shape[1]))])
    return patches, pools


@pytest.mark.gpu
@pytest.mark.parametrize("quality", [5, 50, 75, 92, 100])
@pytest.mark.parametrize("kinds,wild", [((0, 1, 2, 3, 4), False), ((0, 1, 2, 3, 4), True), ((1, 2, 3, 4), False),
                                        ((0, 3), True)])
def test_pruned_selections_equal_scoring_every_candidate(quality, kinds, wild):
    from weft_b200.fit import BatchedFit

    sides = [8, 8, 8, 16, 16, 32, 64]
    patches, pools = _workload(quality + 10 * len(kinds) + wild, sides, kinds, 36, wild)
    extra = _workload(7, sides, kinds, 5, wild)[1]
    caps = [6] * len(sides)

    def reseed(i, patch, pred):
        return list(extra[i])

    want, obj, _ = ofit.greedy_fit(patches, sides, pools, quality, reseed=reseed, caps=caps, max_rounds=3)
    for queue in (True, False):
        fit = BatchedFit(patches, [list(p) for p in pools], quality, caps=caps).use_queue(queue)
        fit.run(reseed=reseed, max_rounds=3)
        assert fit.selected_indices() == want
        np.testing.assert_allclose(fit.objectives(), obj, rtol=1e-5, atol=1e-9)


@pytest.mark.gpu
@pytest.mark.parametrize("quality", [50, 75, 92])
def test_rounds_on_the_device_skip_only_rejected_candidates(quality):
    """Inside one weftk_fit_run a stalled tile's old candidates are not scored again; the host-driven
    rounds score them.  Same selections, objectives, rounds and flags."""
    from weft_b200.fit import BatchedFit

    sides = [8] * 12 + [16] * 6 + [32] * 3 + [64]
    patches, pools = _workload(quality, sides, (0, 1, 2, 3, 4), 60, False)
    fit = BatchedFit(patches, pools, quality, caps=[8] * len(sides))
    fit.run()
    sel, obj, rounds, flags = fit.selected_indices(), fit.objectives(), fit.stats.rounds, fit.t_flags.cpu().numpy()
    assert fit.stats.reseeds > 0
    fit.reset()
    fit.run_device()
    assert fit.selected_indices() == sel and fit.control()["rounds"] == rounds
    np.testing.assert_array_equal(fit.objectives(), obj)
    np.testing.assert_array_equal(fit.t_flags.cpu().numpy() & 1, flags & 1)
    assert int(fit.t_flags.max()) < 8  # no internal marks left behind


def _bound(c, s, comp, src):
    """The kernels' lower bound on a curve's squared error, restated in float32."""
    f = np.float32
    ax, ay, cx, cy, bx, by = (f(v) for v in c.geom[:6])
    px, py, rx, ry = f(0.5) * (ax + cx), f(0.5) * (ay + cy), f(0.5) * (cx + bx), f(0.5) * (cy + by)
    mx, my = f(0.5) * (px + rx), f(0.5) * (py + ry)
    e = f(1e-3) + f(1e-3) * (abs(ax - 2 * cx + bx) + abs(ay - 2 * cy + by))
    y, x = np.meshgrid(np.arange(s, dtype=f) + f(0.5), np.arange(s, dtype=f) + f(0.5), indexing="ij")

    def d2(x0, x1, y0, y1):
        dx = np.maximum(np.maximum(x0 - e - x, x - x1 - e), 0)
        dy = np.maximum(np.maximum(y0 - e - y, y - y1 - e), 0)
        return dx * dx + dy * dy

    d = np.minimum(d2(min(ax, px, mx), max(ax, px, mx), min(ay, py, my), max(ay, py, my)),
                   d2(min(bx, rx, mx), max(bx, rx, mx), min(by, ry, my), max(by, ry, my)))
    sigma = max(0.5, c.geom[6])
    top = np.exp(d * f(-1.0 / (2 * sigma * sigma))) * f(min(max(c.alpha, 0.0), 1.0)) * f(1.0001)
    v, u = src - comp, np.array(c.color0, f) - comp
    uu, uv = (u * u).sum(-1) + f(1e-12), (u * v).sum(-1)
    w = np.minimum(np.maximum(uv / uu, 0), top)
    return float(((v - w[..., None] * u) ** 2).sum())


@pytest.mark.parametrize("s", [8, 16, 32, 64])
def test_curve_bound_is_below_the_curves_error(s):
    rng = np.random.default_rng(s)
    src = rng.random((s, s, 3)).astype(np.float32)
    from weft_b200.candidates import Cand

    for k in range(60):
        c = _cand(rng, 3, s, k % 3 == 0)
        c = Cand(3, c.geom, tuple(float(np.float32(v)) for v in rng.random(3)), None, c.alpha)
        under = [Cand(0, (), tuple(float(v) for v in rng.random(3)), None, 1.0)] if k % 2 else []
        comp = orender.render_tile(under, s) if under else np.zeros((s, s, 3), np.float32)
        err = float(((np.asarray(orender.render_tile(under + [c], s), np.float64) - src) ** 2).sum())
        low, n = _bound(c, s, comp, src), 3.0 * s * s
        assert low * 0.9995 - 4e-6 * np.sqrt(n * low) - 1e-9 <= err, (k, low, err)
