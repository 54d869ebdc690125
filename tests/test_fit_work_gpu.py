"""The work counters name the candidate-pixels that were evaluated: what left an error in the scratch."""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_fit_pruning import _workload

pytestmark = pytest.mark.gpu

OPS = {0: 10, 1: 24, 2: 28, 3: 509, 4: 26}  # FP32 operations per pixel of a kind, and 9 for the error


@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("queue", [True, False])
def test_counters_leave_out_what_a_bound_rejects(queue, variant):
    """Round by round: a candidate's blocks of at most 1024 pixels count where their error is finite, and
    not where the curve's bound left infinity or nothing was written."""
    import torch

    from weft_b200.fit import FIT_INIT, FIT_ROUND, BatchedFit

    sides = [8] * 12 + [16] * 6 + [32] * 3 + [64] * 2
    patches, pools = _workload(3, sides, (0, 1, 2, 3, 4), 60, False)
    fit = BatchedFit(patches, pools, 75, caps=[8] * len(sides)).use_queue(queue)
    fit.configure(variants={8: variant, 16: variant, 32: variant})
    fit.reset()
    tile = np.repeat(np.arange(fit.n), fit.pool_cap)
    px = np.minimum(fit.sizes[tile].astype(np.int64) ** 2, 1024)
    rejected, px0, ops0 = 0, 0, 0
    for mode in (FIT_INIT, FIT_ROUND, FIT_ROUND, FIT_ROUND):
        fit.t_partial.fill_(float("nan"))
        torch.cuda.synchronize()
        fit._round(mode)
        partial = fit.t_partial.cpu().numpy().reshape(-1, 4)
        kinds = fit.t_kind.cpu().numpy()
        blocks = np.isfinite(partial).sum(1)
        rejected += int(np.isinf(partial).sum())
        ops = np.array([OPS.get(int(k), 0) for k in kinds]) + 9
        px0 += int((blocks * px).sum())
        ops0 += int((blocks * px * ops).sum())
        assert fit.work_counters() == (px0, ops0), mode
    assert rejected > 0  # the bound was met
