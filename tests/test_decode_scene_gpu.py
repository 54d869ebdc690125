"""``decode_file`` on the device against the host parser (``_decode_general``): the same pixels, bit for
bit, over every primitive kind, deep and empty stacks, chunk lengths, residual layers, scaled targets and
the raster branch; and the same refusal, or the same pixels, for files with a byte changed."""

from __future__ import annotations

import numpy as np
import pytest

from weft_b200 import bitstream, encode
from weft_b200.candidates import Cand


class _Tile:
    def __init__(self, x, y, size):
        self.x, self.y, self.size = x, y, size


LENGTHS = {0: 0, 1: 4, 2: 5, 3: 7, 4: 6}


def _prim(rng, kind):
    if kind == 5:
        return Cand(5, tuple(rng.random(48)), (0.0, 0.0, 0.0), None, 1.0)
    g = rng.random(LENGTHS[kind]) * 15.0
    if kind in (2, 3):
        g[-1] = rng.random() * 4.0
    return Cand(kind, tuple(g), tuple(rng.random(3)), tuple(rng.random(3)) if kind == 1 else None, rng.random())


def _file(seed, sides, depth, res0=True, res1=True, chunk_tiles=64, same=False):
    rng = np.random.default_rng(seed)
    tiles, x, y, row = [], 0, 0, 0
    for s in sides:
        if x + s > 160:
            x, y, row = 0, y + row, 0
        tiles.append(_Tile(x, y, s))
        x, row = x + s, max(row, s)
    stacks = []
    for _ in sides:
        n = int(rng.integers(0, depth + 1))
        kinds = rng.integers(0, 5, n) if n != 1 else rng.integers(0, 6, 1)
        stacks.append([_prim(rng, 0 if same else int(k)) for k in kinds])
    if same:  # bytes with one dominant symbol
        stacks = [[Cand(0, (), (0.5, 0.5, 0.5), None, 1.0)] for _ in sides]
    n = len(sides)
    return bitstream.encode_weft(160, y + row, 75, tiles, stacks,
                                 rng.integers(-40, 41, (n, 3)).tolist() if res0 else None,
                                 list(rng.integers(-60, 61, (n, 4, 4, 3)).astype(np.int8)) if res1 else None,
                                 chunk_tiles)


SIDES = [8, 16, 32, 64, 8, 8, 16, 32]


def test_layout_takes_ordinary_files_only():
    blob = _file(1, SIDES, 3)
    f, dct, w, h = bitstream.scene_layout(blob)
    assert (f.n_tiles, f.n_res1, f.n_chunks, dct) == (8, 8, 1, None) and w == 160
    assert bitstream.scene_layout(bytearray(blob)) is None
    for cut in (0, 11, 40, len(blob) // 2, len(blob) - 1):
        assert bitstream.scene_layout(blob[:cut]) is None
    for tag in (b"CIDX", b"QTRE", b"HEAD"):
        at = blob.index(tag)
        assert bitstream.scene_layout(blob[:at] + b"XXXX" + blob[at + 4:]) is None


def _on_device(blob, tw=None, th=None):
    scene = bitstream.scene_layout(blob)
    return None if scene is None else encode._decode_on_device(blob, scene, tw, th)


def _covered_once(blob, tw, th):
    """Pixels that at most one tile draws: where rects of less than a pixel share one, either decoder draws
    them in no order."""
    from weft_b200 import render

    wf = bitstream.decode_weft(blob)
    ew, eh = int(wf.meta.get("encode_width", wf.width)), int(wf.meta.get("encode_height", wf.height))
    hits = np.zeros((th, tw), np.int64)
    for t in wf.qtree:
        x, y, w, h = render.tile_rect(*t, tw / ew, th / eh, (tw, th) != (ew, eh))
        hits[y:y + h, x:x + w] += 1
    return hits <= 1


@pytest.mark.gpu
@pytest.mark.parametrize("target", [(None, None), (160, 96), (321, 250), (80, 47), (1, 1)])
@pytest.mark.parametrize("case", [
    dict(seed=2, sides=SIDES, depth=3), dict(seed=3, sides=SIDES * 20, depth=48), dict(seed=4, sides=[8], depth=1),
    dict(seed=5, sides=SIDES * 9, depth=1, res1=False), dict(seed=6, sides=[8] * 200, depth=2, res0=False, res1=False),
    dict(seed=7, sides=SIDES * 5, depth=4, chunk_tiles=1), dict(seed=8, sides=[8] * 700, depth=1, chunk_tiles=700),
    dict(seed=9, sides=[8] * 300, depth=1, chunk_tiles=128, same=True),
])
def test_device_decode_equals_host_parser(case, target):
    blob = _file(**case)
    got = _on_device(blob, *target)
    want = encode._decode_general(blob, *target)
    assert got is not None and got.shape == want.shape
    once = _covered_once(blob, want.shape[1], want.shape[0])
    np.testing.assert_array_equal(got[once], want[once])


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["a", "b"])
def test_device_decode_of_the_raster_branch(golden, which):
    blob = golden("container_dct.npz")[f"file_{which}"].tobytes()
    for target in ((None, None), (200, 150), (50, 37)):
        got = _on_device(blob, *target)
        assert got is not None
        np.testing.assert_array_equal(got, encode._decode_general(blob, *target))


@pytest.mark.gpu
@pytest.mark.parametrize("part", ["PRIM", "CIDX", "TOC ", "QTRE", "RES0", "any"])
def test_changed_bytes_end_as_with_the_host_parser(part):
    blob = _file(11, SIDES * 4, 3, chunk_tiles=8)
    spans, _ = bitstream._directory(blob)
    at, ln = (0, len(blob)) if part == "any" else spans[part.encode()]
    rng = np.random.default_rng(len(part) + at)
    for _ in range(40):
        bad = bytearray(blob)
        where = at + int(rng.integers(ln))
        bad[where] ^= int(rng.integers(1, 256 if part != "TOC " else 16))
        bad = bytes(bad)

        def outcome(f):
            try:
                return f(bad, 64, 48)
            except Exception as e:  # noqa: BLE001 - the refusal itself is compared
                return f"{type(e).__name__}: {e}"

        got, want = outcome(encode.decode_file), outcome(encode._decode_general)
        if isinstance(want, str):
            assert got == want
        else:
            once = _covered_once(bad, 64, 48)
            np.testing.assert_array_equal(got[once], want[once])
