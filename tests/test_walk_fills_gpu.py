"""The decoder walk's fills (lone constant layers) against its per-pixel kernel: the same constant with a
second layer of alpha 0 above it, which leaves every bit as it is but goes through the other kernel.  Rows
with and without 16-byte alignment, rects cut by every edge and narrower than a slot, with and without RES1
grids, and lists long enough that warps take several items."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _walk(descs, prims, grids, h, w, pad):
    import torch

    from weft_b200 import _lib, render

    items = render.decode_items(descs, h, w, prims)
    dev = [torch.from_numpy(a).cuda() for a in (descs.view(np.uint8), items, prims.view(np.uint8), grids)]
    buf = torch.full((h * w * 3 + 4,), -1.0, dtype=torch.float32, device="cuda")
    out = buf[pad:pad + h * w * 3]
    lib = _lib.lib_for_device(0)
    rc = lib.weftk_render_tiles(_lib.ptr(dev[0]), len(descs), _lib.ptr(dev[1]), len(items), _lib.ptr(dev[2]), 0, 0,
                                _lib.ptr(dev[3]) if len(grids) else 0, len(grids), _lib.ptr(out), h, w, 0,
                                torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    return buf.cpu().numpy()


@pytest.mark.parametrize("w", [64, 61, 1, 3])
@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("many", [False, True])
def test_fills_equal_the_general_kernel(w, pad, residual, many):
    from weft_b200._lib import PRIM_DTYPE, TILE_DECODE_DTYPE

    rng = np.random.default_rng(w + pad)
    h = 2400 if many else 75
    rects, y = [], -5
    sides = [1, 2, 3, 5, 8, 13, 30, 64]
    while y < h:
        s, x = sides[len(rects) % len(sides)], -2
        while x < w:
            rects.append((x, y, sides[int(rng.integers(len(sides)))], s))
            x += rects[-1][2]
        y += s
    n = len(rects)
    d = np.zeros(n, TILE_DECODE_DTYPE)
    for k, f in enumerate(("target_x0", "target_y0", "target_w", "target_h")):
        d[f] = [r[k] for r in rects]
    d["source_size"] = 8
    d["res1_index"] = rng.integers(-1, 5, n) if residual else -1
    for f in ("res0_r", "res0_g", "res0_b"):
        d[f] = rng.integers(-30, 31, n) / np.float32(255.0)
    prims = np.zeros(2 * n, PRIM_DTYPE)
    prims["color0"] = rng.random((2 * n, 3))
    prims["alpha"][0::2] = rng.random(n)
    d["prim_offset"] = 2 * np.arange(n)
    grids = (rng.random((5 if residual else 0, 48)) - 0.5).astype(np.float32)
    d["prim_count"] = 1
    fills = _walk(d, prims, grids, h, w, pad)
    d["prim_count"] = 2
    np.testing.assert_array_equal(fills, _walk(d, prims, grids, h, w, pad))
    assert (fills >= 0).sum() == h * w * 3
