"""Rules of the kernels' sources that no run shows reliably: breaking them gives a fault only where a warp's lanes drift apart or a launch
overlaps its predecessor."""
import glob
import os
import re

from _support import ROOT

CSRC = os.path.join(ROOT, "gretacore-v3_b200", "csrc")


def _blocks(text, head):
    """The brace blocks that follow matches of `head`."""
    for m in re.finditer(head, text):
        depth = 0
        for i in range(m.end() - 1, len(text)):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            if depth == 0:
                yield text[m.end():i]
                break


def _code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def test_raw_weights_are_given_back_behind_their_use():
    """The dequantising warps let the next copy into a raw unit once its values have been stored to tensor memory, not once the loads are issued."""
    text = _code(os.path.join(CSRC, "gemm_ts.cu"))
    assert text.count("mbar_arrive(&raw_empty[slot])") == 1
    assert text.index("tmem_st_wait();") < text.index("mbar_arrive(&raw_empty[slot])")
