"""What the DCT kernel reads two doubles at a time is declared with the alignment that takes."""

from __future__ import annotations

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "weft_b200", "csrc")


def test_arrays_read_as_double2_are_aligned():
    with open(os.path.join(CSRC, "weftk_dct.cu")) as f:
        text = f.read()
    read = set(re.findall(r"reinterpret_cast<(?:const )?double2\*>\((g_\w+)", text))
    assert read  # the table the kernel copies
    for name in read:
        assert re.search(rf"__device__ __align__\(16\) double {name}\[", text), name
    for declared in re.findall(r"extern __shared__ ([^;]*)\bdouble \w+\[\];", text):
        assert "__align__(16)" in declared
