"""The raster branch at the sizes where its kernels change course: a DCT layer's classes of tiles
(partly filled CTAs, every side, launches that follow one another, tiles smaller than their class), and
the resize's window in shared memory (widths with and without four-wide stores, one-pixel sides,
downscales that take fewer rows per CTA and ones that fall back to two kernels)."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layer(sides, chroma, band, seed):
    """Tiles in a strip, their descriptors and coefficients, and each tile's own stream."""
    from weft_b200.raster import DCT_TILE_DTYPE

    rng = np.random.default_rng(seed)
    descs = np.zeros(len(sides), DCT_TILE_DTYPE)
    x, stream, base = 0, [], 0
    for t, s in enumerate(sides):
        descs[t]["x"], descs[t]["y"], descs[t]["size"] = x, 3 * (t % 4), s
        descs[t]["step_scale"] = 1.0 + 0.25 * (t % 3)
        for c in range(3):
            n = s // 2 if chroma == 2 and c else s
            descs[t]["coef_base"][c], descs[t]["coef_stride"][c] = base, 1 + (t % 2)
            q = np.zeros(n * n * (1 + (t % 2)), np.int16)
            q[:: 1 + (t % 2)] = np.round(rng.laplace(0.0, 3.0, n * n)).astype(np.int16)
            stream.append(q)
            base += len(q)
        x += s
    return descs, np.concatenate(stream), x


def _run(descs, coeffs, groups, chroma, band, image):
    import torch

    from weft_b200 import _lib

    lib = _lib.lib_for_device(0)
    td = torch.from_numpy(descs.view(np.uint8)).cuda()
    tc = torch.from_numpy(coeffs).cuda()
    st = ctypes.c_int(0)
    lib.weftk_device_status(ctypes.addressof(st))
    for side, first, count in groups:
        rc = lib.weftk_dct_apply(_lib.ptr(td) + first * descs.itemsize, count, _lib.ptr(tc), len(coeffs), chroma, band,
                                 0.02, 4.0, side, _lib.ptr(image), int(image.shape[1]), int(image.shape[0]), 0,
                                 torch.cuda.current_stream().cuda_stream)
        assert rc == 0
    _lib.check(lib.weftk_device_status(ctypes.addressof(st)), "weftk_device_status")
    assert st.value == 0
    return image


@pytest.mark.parametrize("chroma", [0, 1, 2])
@pytest.mark.parametrize("band", [0, 1])
@pytest.mark.parametrize("counts", [(1, 1, 1, 1, 1), (257, 65, 17, 5, 2), (0, 64, 0, 4, 0)])
def test_dct_classes(chroma, band, counts):
    import torch

    from oracle import dct as odct

    sides = [s for s, n in zip((4, 8, 16, 32, 64), counts) for _ in range(n)]
    descs, coeffs, width = _layer(sides, chroma, band, sum(counts) + chroma)
    height = 70  # the tall tiles' last rows stay inside, the strip's right edge is cut
    rng = np.random.default_rng(1)
    base = rng.random((height, width - 3, 3), dtype=np.float32)
    groups, at = [], 0
    for s, n in zip((4, 8, 16, 32, 64), counts):
        groups.append((s, at, n))
        at += n
    got = _run(descs, coeffs, groups, chroma, band, torch.from_numpy(base.copy()).cuda()).cpu().numpy()
    # every tile listed in the largest class: smaller tiles than their class, the same values
    one = _run(descs, coeffs, [(64, 0, len(sides))], chroma, band, torch.from_numpy(base.copy()).cuda()).cpu().numpy()
    np.testing.assert_array_equal(got, one)

    want, largest = base.astype(np.float64), 0.0
    m = np.array([[1.0, 0.0, 1.402], [1.0, -0.344136, -0.714136], [1.0, 1.772, 0.0]])
    for d in descs:
        s, planes = int(d["size"]), []
        for c in range(3):
            n = s // 2 if chroma == 2 and c else s
            order = odct.zigzag(n) if band else np.arange(n * n)
            pos = np.empty(n * n, np.int64)
            pos[order] = np.arange(n * n)
            q = coeffs[d["coef_base"][c] + pos * d["coef_stride"][c]].astype(np.float64).reshape(n, n)
            k = np.arange(n)
            step = float(np.float32(0.02)) * (1.5 if chroma and c else 1.0) * d["step_scale"]
            q = q * (step * (1.0 + 4.0 * (k[:, None] + k[None, :]) / (2.0 * (n - 1))))
            a = odct.idct_matrix(n)
            p = (a.T @ q @ a).astype(np.float32).astype(np.float64)
            largest = max(largest, float(np.abs(p).max()))
            planes.append(np.repeat(np.repeat(p, s // n, 0), s // n, 1))
        rgb = np.stack(planes, -1)
        if chroma:
            rgb = rgb @ m.T
        x, y = int(d["x"]), int(d["y"])
        h, w = min(s, height - y), min(s, base.shape[1] - x)
        want[y:y + h, x:x + w] = np.clip(want[y:y + h, x:x + w] + rgb[:h, :w], 0.0, 1.0)
    # a plane's float32 value may be the neighbouring one (weights 1 and 1.772 at most); the residual and
    # the sum, at most 1 where the clip does not hide it, are rounded once each
    tol = 2.8 * float(np.spacing(np.float32(largest))) + 2.0 ** -23
    assert float(np.max(np.abs(got - want))) <= tol


@pytest.mark.parametrize("size,target", [
    ((129, 65), (128, 64)), ((64, 48), (256, 130)), ((64, 48), (257, 129)), ((1, 1), (5, 3)), ((33, 1), (12, 1)),
    ((1, 40), (3, 7)), ((300, 211), (131, 97)), ((500, 400), (132, 101)), ((700, 900), (100, 90)),
    ((1200, 90), (60, 400)), ((90, 1200), (400, 60)), ((1500, 1100), (48, 20)), ((640, 360), (640, 720)),
])
def test_resize_windows(size, target):
    import torch

    from oracle import dct as odct
    from weft_b200 import raster

    (w, h), (tw, th) = size, target
    rng = np.random.default_rng(w * 7 + th)
    img = (rng.random((h, w, 3), dtype=np.float32) * np.float32(1.2) - np.float32(0.1))
    got = raster.resize(torch.from_numpy(img).cuda(), tw, th).cpu().numpy()
    u8 = np.clip(img * np.float32(255.0), 0.0, 255.0).astype(np.uint8)
    want = odct.resize_bilinear_u8(u8, tw, th).astype(np.float32) / np.float32(255.0)
    np.testing.assert_array_equal(got, want)
