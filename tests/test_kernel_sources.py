"""Rules of the kernels' sources that no run shows reliably: breaking them gives a fault only where a warp's lanes drift apart or a launch
overlaps its predecessor."""
import glob
import os
import re

import pytest

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


ELECTING = [os.path.basename(p) for p in sorted(glob.glob(os.path.join(CSRC, "*.cu"))) if "elect_one()" in _code(p)]


@pytest.mark.parametrize("name", ELECTING)
def test_lanes_of_an_issuing_warp_meet_between_wait_and_issue(name):
    """All lanes of an issuing warp wait on a barrier's parity and one issues.  A lane still waiting when the issue lets the barrier move on two
    phases would read it as not yet done, run into the time limit and abort the kernel: every wait is followed by __syncwarp(), and every
    lane reaches it (no way out of the loop in between)."""
    text = _code(os.path.join(CSRC, name))
    roles = [b for b in _blocks(text, r"if \(warp == \d\) \{") if "leader" in b]
    assert len(roles) >= 2 and text.count("elect_one()") * 2 <= len(roles)
    for body in roles:
        assert len(re.findall(r"if \(ok\) ok = mbar_wait\([^;]*;\s*__syncwarp\(\);", body)) == len(re.findall(r"ok\w* = mbar_wait|!mbar_wait", body)) > 0
        assert "break" not in body and not re.search(r"for \([^{]*\bok\b[^{]*\{", body)
        # copies are counted by the lane that issued them
        assert len(re.findall(r"if \(leader && \*abort_flag\) drain_copies\(", body)) == body.count("drain_copies(")
