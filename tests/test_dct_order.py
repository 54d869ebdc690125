"""A DCT layer's launches are ordered behind whatever writes their inputs: only the further tile sides of
one layer may start beside the launch before them."""

from __future__ import annotations

import numpy as np
import pytest

from weft_b200 import _lib, raster


def _block(sides, seed):
    """A tile-major 4:2:0 block over a strip of tiles of the given sides, and the tiles."""
    rng = np.random.default_rng(seed)
    x = np.concatenate([[0], np.cumsum(sides)])[:-1]
    n = sum(s * s + 2 * (s // 2) ** 2 for s in sides)
    q = np.round(rng.laplace(0.0, 3.0, n)).astype(np.int16)
    return raster.DctBlock(q, 0.02, 3, 4.0, 2, b"", 0, 0, b""), [(int(a), 0, int(s)) for a, s in zip(x, sides)]


class _Layouts:
    """Records the layout argument of each call."""

    def __init__(self):
        self.layouts = []

    def weftk_dct_apply(self, *args):
        if args[1]:
            self.layouts.append(args[5])
        return 0


@pytest.mark.parametrize("sides,want", [((8,), [0]), ((16, 16), [0]), ((8, 16, 64), [0, 0x100, 0x100])])
def test_only_a_layers_further_launches_may_overlap(sides, want):
    layer = object.__new__(raster.DctLaunch)
    layer.block, tiles = _block(sides, 1)
    layer.descs = raster.tile_table(layer.block, tiles, sum(sides), 64)
    layer.width, layer.height, layer.lib = sum(sides), 64, _Layouts()
    layer.t_coeffs, layer.t_descs = layer.block.coeffs, layer.descs.view(np.uint8)
    side = layer.descs["size"]
    layer.groups = [(int(v), int(np.searchsorted(side, v, "left")), int(np.searchsorted(side, v, "right")))
                    for v in np.unique(side)]
    for _ in range(2):  # the next pass over the same layer starts in order again
        layer.lib.layouts.clear()
        layer.run(np.zeros((64, sum(sides), 3), np.float32), 0)
        assert layer.lib.layouts == want


@pytest.mark.parametrize("layout", [2, 3, -1, 0x100 | 2, 0x200, 0x80])
def test_other_layout_values_stay_refused(layout):
    img = np.zeros(3, np.float32)
    rc = _lib.load().weftk_dct_apply(0, 0, 0, 0, 2, layout, 0.01, 0.0, 16, _lib.ptr(img), 1, 1, 0, 0)
    assert rc == -1 and "layout" in _lib.last_error()


@pytest.mark.gpu
@pytest.mark.parametrize("sides", [(8,), (64, 32, 16, 8), (4, 8, 8, 16, 16, 32, 64)])
def test_inputs_written_by_a_kernel_just_before(sides):
    """Descriptors and coefficients filled by kernels on the stream directly before the layer, twice
    with different values: the same image as from arrays that were copied beforehand."""
    import torch

    want, layers = [], []
    base = np.random.default_rng(5).random((64, sum(sides), 3), dtype=np.float32)
    for seed in (2, 3):
        block, tiles = _block(sides, seed)
        layers.append(raster.DctLaunch(block, tiles, sum(sides), 64))
        img = torch.from_numpy(base.copy()).cuda()
        layers[-1].run(img, torch.cuda.current_stream().cuda_stream)
        want.append(img.cpu().numpy())
    late, _ = _block(sides, 4)
    late = raster.DctLaunch(late, tiles, sum(sides), 64)
    images = [torch.from_numpy(base.copy()).cuda() for _ in range(2)]
    big = torch.zeros(1 << 24, device="cuda")
    torch.cuda.synchronize()
    for img, layer in zip(images, layers):
        big.add_(1.0)  # keeps the stream busy while what follows is enqueued
        late.t_descs.zero_()
        torch.add(layer.t_descs, 0, out=late.t_descs)
        torch.add(layer.t_coeffs, 0, out=late.t_coeffs)
        late.run(img, torch.cuda.current_stream().cuda_stream)
    for img, w in zip(images, want):
        np.testing.assert_array_equal(img.cpu().numpy(), w)
