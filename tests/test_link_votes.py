"""Votes of the link gather (csrc/lbm_linkgather.cuh): which lanes are together at a point
is not fixed, so a vote over the active lanes may choose between two codes that both serve
the lane, but no value or address may depend on it.  Source check: no GPU."""
import os
import re

from taichi_lbm3d_gb300 import build


def test_only_the_choice_of_code_asks_the_active_lanes():
    txt = open(os.path.join(build.CSRC, "lbm_linkgather.cuh")).read()
    code = re.sub(r"//[^\n]*", "", txt)
    asks = [line for line in code.splitlines() if "__activemask" in line]
    assert len(asks) == 1 and "any_record() const" in asks[0]
    assert "__all_sync" not in code and "__ballot_sync" not in code
