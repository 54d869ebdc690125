"""Device quadtree tiling and extraction against the host's over the shapes where the kernels divide their
work: one macro tile, sides that cut macro tiles, every ratio of largest to smallest tile, more macro
tiles than one scan step of a placement CTA.  Lists are equal tile for tile, pixels bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,max_tile,min_tile", [
    (1, 1, 64, 8), (64, 64, 64, 8), (65, 63, 64, 8), (300, 129, 64, 16), (200, 200, 64, 32), (257, 65, 64, 64),
    (100, 77, 32, 8), (90, 40, 16, 8), (33, 50, 16, 16), (1111, 1100, 8, 8), (700, 520, 64, 8),
])
def test_tiles_equal_the_host_decomposition(w, h, max_tile, min_tile):
    import torch

    from weft_b200 import frontend, quadtree
    from weft_b200.synth import make_image_u8, srgb_u8_to_linear

    u8 = make_image_u8(w, h, 60, 4) if min(w, h) > 16 else np.full((h, w, 3), 90, np.uint8)
    img = srgb_u8_to_linear(u8)
    host_tiles = quadtree.decompose(img, rule="variance", threshold=100.0, min_tile=min_tile, max_tile=max_tile,
                                    image_u8=u8)
    want = [(t.x, t.y, t.size) for t in host_tiles]
    d_img = torch.from_numpy(u8).cuda()
    tiles, count = frontend.decompose_device(d_img, 100.0, min_tile=min_tile, max_tile=max_tile)
    got = tiles.cpu().numpy()
    assert count == len(want)
    np.testing.assert_array_equal(got, np.array(want, np.int32))
    src4, _ = frontend.extract_device(d_img, tiles, got[:, 2].copy())
    host = np.concatenate([p.reshape(-1, 3) for p in quadtree.extract_tiles(img, host_tiles, max_tile)])
    np.testing.assert_array_equal(src4[:, :3].cpu().numpy(), host)
