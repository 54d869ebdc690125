"""What a large file's decode takes on the device is given back when the call returns."""

from __future__ import annotations

import struct

import numpy as np
import pytest

from weft_b200 import bitstream, encode
from weft_b200.candidates import Cand


class _Tile:
    def __init__(self, x, y, size):
        self.x, self.y, self.size = x, y, size


def _file(monkeypatch, n, layers):
    """A file of n tiles of 8 px, each with the same stack; chunks stored, not entropy-coded."""
    tiles = [_Tile(8 * (i % 200), 8 * (i // 200), 8) for i in range(n)]
    stack = [Cand(0, (), (0.25, 0.5, 0.75), None, 0.5)] * layers
    part, _ = bitstream.encode_tiles([stack])
    monkeypatch.setattr(bitstream, "encode_tiles", lambda s: (part * n, [len(part) * i for i in range(n + 1)]))
    monkeypatch.setattr(bitstream, "encode_bytes", lambda b: b"\0" + struct.pack("<I", len(b)) + b)
    blob = bitstream.encode_weft(1600, 8 * (-(-n // 200)), 75, tiles, [stack] * n)
    monkeypatch.undo()
    return blob


@pytest.mark.gpu
def test_large_files_leave_no_large_buffers(monkeypatch):
    import torch

    small, large = _file(monkeypatch, 400, 1), _file(monkeypatch, 30000, 48)
    assert len(large) > 10_000_000
    first = encode.decode_file(small)
    free = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        out = encode.decode_file(large)
    # the image's own buffer stays: 1600 x 1200 x 12 bytes and a quarter more, 27 MiB
    assert free - torch.cuda.mem_get_info()[0] <= 64 << 20
    scene = bitstream.scene_layout(large)
    assert scene is not None and encode._decode_on_device(large, scene, None, None) is not None
    assert out.shape == (1200, 1600, 3) and np.all(out == out[0, 0])
    np.testing.assert_array_equal(encode.decode_file(small), first)
