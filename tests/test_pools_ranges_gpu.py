"""The device pool generator where its short cuts end: de-duplication keys whose colours leave the
packed range (and the mixture with ones that stay in it), negative and signed-zero pixels, single
bright pixels (regions of one pixel, empty sides), gradients along one axis (every angle in one
histogram bin: the longest pairwise sum) and along the diagonals (every angle off the axes).  The
pools equal the host restatement's record for record, so there is no tolerance."""

from __future__ import annotations

import numpy as np
import pytest

from test_pools_gpu import _compare

pytestmark = pytest.mark.gpu


def _patches(side, kind):
    rng = np.random.default_rng(side + 1000 * len(kind))
    y, x = np.mgrid[0:side, 0:side].astype(np.float32)
    if kind == "out_of_range":
        wide = (rng.random((side, side, 3), dtype=np.float32) - np.float32(0.5)) * np.float32(90.0)
        half = rng.random((side, side, 3), dtype=np.float32)
        half[:, : side // 2] += np.float32(35.0)
        step = np.full((side, side, 3), 40.0, np.float32)
        step[side // 2:] = -40.0
        return [wide, half, step]
    if kind == "signed":
        zeros = np.where(rng.random((side, side, 3)) < 0.5, np.float32(0.0), np.float32(-0.0)).astype(np.float32)
        return [zeros, -rng.random((side, side, 3), dtype=np.float32)]
    if kind == "one_pixel":
        out = []
        for at in ((0, 0), (side - 1, side - 1), (side // 2, side // 2 - 1)):
            p = np.zeros((side, side, 3), np.float32)
            p[at] = 1.0
            out.append(p)
        return out
    ramps = {"axis": (x, y), "diagonal": (x + y, side + x - y, 3 * x + y)}[kind]
    return [np.repeat((r / np.float32(4 * side))[:, :, None], 3, axis=2).astype(np.float32) for r in ramps]


@pytest.mark.parametrize("side", [8, 16, 32, 64])
@pytest.mark.parametrize("kind", ["out_of_range", "signed", "one_pixel", "axis", "diagonal"])
def test_pools_outside_the_ordinary_range(side, kind):
    bad, n = _compare(_patches(side, kind), 75)
    assert n > 0 and not bad, bad
