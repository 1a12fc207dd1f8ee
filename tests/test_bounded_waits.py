"""Bounded waits in kernels whose loops depend on them (no GPU needed: the source is read)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kyojin_mac_b200", "csrc")


def test_prefill_waits_are_warp_votes():
    """The decoders of the prefill GEMM leave their loop when a wait gives up, and the loop body is full of warp-wide instructions: a wait that each lane answers
    for itself would let some lanes leave and the others wait for them for good. So the kernel waits through the vote only."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "gemm_kq.cu")).read())
    vote = re.search(r"bool mbar_wait_warp\(.*\n", text).group(0)
    assert "__all_sync(0xffffffffu, mbar_wait_fast(" in vote
    rest = text.replace(vote, "")
    assert rest.count("mbar_wait_warp(") >= 6 and not re.search(r"mbar_wait_(fast|slow|bounded)\(|mbar_try_wait\(", rest)
