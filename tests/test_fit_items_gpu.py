"""Work items that a caller built wrongly are refused by every scoring launch, with and without the queue."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from tests.test_fit_pruning import _workload

pytestmark = pytest.mark.gpu


def _status(fit):
    from weft_b200 import _lib

    st = ctypes.c_int(0)
    _lib.check(fit.lib.weftk_device_status(ctypes.addressof(st)), "weftk_device_status")
    return st.value


def _round_with(side, variant, queue, mode, item):
    """Device status after a round whose only item is ``item`` (tile, block, first, count)."""
    import torch

    from weft_b200.fit import BatchedFit

    patches, pools = _workload(side, [side], (0, 1, 2, 4), 300, False)
    fit = BatchedFit(patches, pools, 92, caps=[8]).use_queue(queue)
    cls = min(side, 32)
    fit.configure(variants={cls: variant})
    fit.reset()
    if mode:
        fit._round(0)
    _status(fit)
    fit.t_items[cls] = torch.tensor([item], dtype=torch.int32, device=fit.device)
    fit.n_items[cls] = 1
    fit._round(mode)
    return _status(fit)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("queue", [True, False])
@pytest.mark.parametrize("side,variant", [(8, 0), (8, 2), (16, 0), (16, 1), (16, 2), (32, 0), (64, 1), (64, 2)])
@pytest.mark.parametrize("count", [129, 200, 256])
def test_more_candidates_than_an_item_holds(side, variant, queue, mode, count):
    assert _round_with(side, variant, queue, mode, (0, 0, 0, 128)) == 0
    assert _round_with(side, variant, queue, mode, (0, 0, 0, count)) == -1


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("queue", [True, False])
@pytest.mark.parametrize("side,variant", [(8, 0), (8, 2), (16, 0), (16, 1), (32, 0), (64, 1)])
@pytest.mark.parametrize("block", [-1, -4, 4, 1 << 22, (1 << 31) - 1, -(1 << 31)])
def test_blocks_outside_the_tile(side, variant, queue, mode, block):
    """(1 << 22 blocks of 1024 pixels: a product past 32 bits.)"""
    assert _round_with(side, variant, queue, mode, (0, block, 0, 64)) == -1
