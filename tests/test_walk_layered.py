"""The walk of pictures with many evaluated layers: the same image whichever number of places its per-pixel
kernel is given, and the rule that chooses it."""

from __future__ import annotations

import numpy as np
import pytest

from weft_b200 import render
from weft_b200._lib import PRIM_DTYPE, TILE_DECODE_DTYPE


def _scene(counts, kinds, side=16, per_row=40):
    n = len(counts)
    d = np.zeros(n, TILE_DECODE_DTYPE)
    d["prim_count"], d["prim_offset"] = counts, np.concatenate([[0], np.cumsum(counts)[:-1]])
    d["target_x0"], d["target_y0"] = side * (np.arange(n) % per_row), side * (np.arange(n) // per_row)
    d["target_w"] = d["target_h"] = d["source_size"] = side
    d["res1_index"] = -1
    rng = np.random.default_rng(n)
    rec = np.zeros(int(np.sum(counts)), PRIM_DTYPE)
    rec["kind"] = kinds
    rec["geom"], rec["color0"], rec["color1"] = rng.random((len(rec), 7)) * 15, rng.random((len(rec), 3)), rng.random((len(rec), 3))
    rec["alpha"] = rng.random(len(rec))
    return d, rec


@pytest.mark.parametrize("counts,kinds,layered", [
    ([1, 1, 1], [0, 0, 0], 0), ([1, 1, 1], [1, 0, 0], 0), ([1, 1], [1, 0], 1), ([1] * 9 + [4], [0] * 13, 0),
    ([1] * 7 + [4], [0] * 11, 1), ([0, 0], [], 0), ([1] * 3, [5, 5, 0], 1),
])
def test_flag_from_one_evaluated_layer_for_two_tiles(counts, kinds, layered):
    d, rec = _scene(counts, kinds)
    assert render.walk_flags(d, rec) == (render.WALK_LAYERED if layered else 0)


@pytest.mark.gpu
@pytest.mark.parametrize("layers", [1, 2, 24])
@pytest.mark.parametrize("n", [3, 1000])
def test_same_image_with_and_without_the_flag(layers, n):
    import torch

    from weft_b200 import _lib

    rng = np.random.default_rng(layers)
    counts = np.where(rng.random(n) < 0.5, 1, layers)
    d, rec = _scene(counts, rng.integers(0, 5, int(counts.sum())))
    h, w = 16 * (-(-n // 40)), 640
    items = render.decode_items(d, h, w, rec)
    dev = [torch.from_numpy(a).cuda() for a in (d.view(np.uint8), items, rec.view(np.uint8))]
    lib, images = _lib.lib_for_device(0), []
    for flags in (0, render.WALK_LAYERED):
        out = torch.zeros((h, w, 3), device="cuda")
        _lib.check(lib.weftk_render_tiles(_lib.ptr(dev[0]), n, _lib.ptr(dev[1]), len(items), _lib.ptr(dev[2]), 0, 0, 0, 0,
                                          _lib.ptr(out), h, w, flags, torch.cuda.current_stream().cuda_stream), "walk")
        images.append(out.cpu().numpy())
    np.testing.assert_array_equal(images[0], images[1])
    np.testing.assert_array_equal(images[0], render._launch(d, rec, np.zeros((0, 48), np.float32), None, h, w))
