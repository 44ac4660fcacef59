"""Barrier waits of the kernels whose warps go on with warp-wide operations
end the same way for all lanes.  Each lane tries a barrier by itself and gives
up after a limit; a warp that left its loop in part would wait for its own
lanes for good in the next shuffle, so k_ksolve and k_syrk_update take a
wait's result through warp_agree.  (No test can make a lane time out alone;
this one reads the sources.)"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hfls_b200", "csrc", "device")


def body(path, name):
    """Text of the kernel's definition, comments stripped."""
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, path)).read())
    at = next(m.start() for m in re.finditer(r"\b" + name + r"\(", src) if "{" in src[m.start():src.index(";", m.start())])
    depth, i = 0, src.index("{", at)
    for j in range(i, len(src)):
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        if depth == 0:
            return src[i:j]


@pytest.mark.parametrize("path,name,waits", [("ksolve.cu", "k_ksolve", 4), ("setup_kernels.cu", "k_syrk_update", 2)])
def test_lanes_of_a_warp_agree_on_a_wait(path, name, waits):
    text = body(path, name)
    calls = [m.start() for m in re.finditer(r"\b(mbar_wait|bar_wait_cluster)\(", text)]
    assert len(calls) == waits
    for c in calls:
        alone = text[:c].endswith("warp_agree(")
        # lanes waiting for different barriers agree after the loop
        loop = re.match(r"[^;]*;\s*ok = warp_agree\(ok\);", text[c:])
        assert alone or loop, text[c - 60:c + 60]
