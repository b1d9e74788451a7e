"""Tensor-memory loads are instructions of a whole warp.  Where code that runs per
lane comes before them in the analysis kernel (a poll on a barrier, one lane's
chain of loads), the warp is brought together explicitly."""
import re

from conftest import ROOT

CSRC = ROOT / "metada_gb300" / "csrc"


def test_polls_end_with_the_warp_together():
    text = (CSRC / "mg_tf32op.cuh").read_text()
    body = text[text.index("bool wait_one("):]
    body = body[: body.index("\n}")]
    assert body.index("mbar_wait(") < body.index("__syncwarp();") < body.index("tc_fence_after();")


def test_one_lanes_pull_ends_with_the_warp_together():
    text = (CSRC / "mg_letkf_tc.cu").read_text()
    assert re.search(r"if \(tid == kThreads - 1\) pull\(prm, s_it\);\s*__syncwarp\(\);", text)
