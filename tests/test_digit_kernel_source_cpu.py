"""tcgen05.commit tracks the asynchronous operations of the thread that executes
it, so the commits of the digit kernel belong to the lane that issues its MMAs.
The path where this decides (tensor memory freed after a wait ran out) is one
that no test may provoke on a GPU: checked in the source."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gcge_gb300",
                   "csrc", "ozaki_tc.cu")


def test_commits_come_from_the_lane_that_issues_the_mmas():
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    kernel = text[text.index("auto issue_mma"):]
    end = kernel.index("};")
    assert "tc_mma(" in kernel[:end] and "tc_commit(" in kernel[:end]
    uses = re.findall(r"[^\n]*\b(?:issue_mma|tc_commit|tc_mma)\([^\n]*", kernel[end:])
    assert len(uses) >= 2
    assert all(u.strip().startswith("if (tc_elect()) ") for u in uses), uses
