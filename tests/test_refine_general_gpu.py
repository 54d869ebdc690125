"""The general refine kernels at the edges of their tile classes and history depths: tile sides on both
sides of each class boundary, stacks on both sides of each depth, against the float64 restatement."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.test_refine_gpu import F64, _rand_stack, ref_tile_loss

pytestmark = pytest.mark.gpu


def _stacks(sides, depths, soft, seed):
    rng = np.random.default_rng(seed)
    patches = [rng.random((s, s, 3), dtype=np.float32) for s in sides]
    stacks = []
    for s, d in zip(sides, depths):
        st = []
        while len(st) < d:
            st += [p for p in _rand_stack(rng, max(s, 4), 8) if (p.kind == 4) <= soft]
        stacks.append(st[:d])
    return patches, stacks


@pytest.mark.parametrize("residual,sides", [(False, (1, 2, 3, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64)),
                                            (True, (8, 16, 32, 64))])
@pytest.mark.parametrize("depth", [1, 4, 5, 16, 17, 32])
def test_general_loss_and_gradient_match_float64(residual, sides, depth):
    from weft_b200.refine import StackSet

    depths = [max(1, depth - (i % 2)) for i in range(len(sides))]
    patches, stacks = _stacks(sides, depths, False, depth)
    ss, params = StackSet.from_stacks(patches, stacks)
    assert ss.max_prims == depth
    g = torch.rand(ss.n, device=params.device) + 0.5
    got = ss.loss_backward(params, g, residual=residual).cpu().numpy()
    loss = ss.loss(params, residual=residual).cpu().numpy()
    rows, off = params.cpu().numpy().astype(np.float64), ss.prim_off_np
    for t in range(ss.n):
        r = torch.tensor(rows[off[t]:off[t + 1]], dtype=F64, requires_grad=True)
        want = ref_tile_loss(list(r), [p.kind for p in stacks[t]], patches[t], False, residual)
        (want * float(g[t])).backward()
        # float32 forward and sums: the bounds of the existing float64 checks
        assert loss[t] == pytest.approx(float(want.detach()), rel=1e-4, abs=1e-7)
        w = r.grad.numpy()[:, :14]
        scale = max(np.abs(w).max(), 1e-5)
        assert np.abs(got[off[t]:off[t + 1], :14] - w).max() / scale < 2e-3, (sides[t], depths[t])


@pytest.mark.parametrize("residual", [False, True])
def test_general_split_does_not_change_results(residual):
    """Without an order every tile finds its own class; tiles listed in another class (more or fewer
    warps) give the same losses and gradients up to the order of their sums."""
    from weft_b200.refine import StackSet

    sides = (8, 64, 16, 32, 8, 64, 32, 16)
    patches, stacks = _stacks(sides, [3] * len(sides), True, 5)
    ss, params = StackSet.from_stacks(patches, stacks)
    g = torch.rand(ss.n, device=params.device) + 0.5

    def both():
        return ss.loss(params, residual=residual), ss.loss_backward(params, g, residual=residual)

    want = both()
    splits = [("none", None, (0, 0, 0)), ("all big", ss.st.order, (ss.n, 0, 0)), ("all mid", ss.st.order, (0, ss.n, 0)),
              ("all 16", ss.st.order, (0, 0, ss.n)), ("all small", ss.st.order, (0, 0, 0))]
    for name, order, (a, b, c) in splits:
        ss.st.order, ss.st.n_big, ss.st.n_mid, ss.st.n_s16 = order, a, b, c
        got = both()
        for x, y in zip(got, want):
            assert float((x - y).abs().max()) <= 2e-5 * float(y.abs().max()), name
