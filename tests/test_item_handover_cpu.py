"""Hand-over of work items to a running CTA (csrc/fwd.cu, csrc/bwd.cu): a wait that has run out is never taken for an item."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sageattention_b200", "csrc")


@pytest.mark.parametrize("name", ["fwd.cu", "bwd.cu"])
def test_an_expired_hand_over_is_looked_at(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    calls = re.findall(r"^.*mbar_wait_item\w*\(.*$", text, re.M)
    assert len(calls) == 6
    for line in calls:      # its answer ends the loop over the items, or the producer's search for one
        assert re.search(r"if \(!mbar_wait_item\w*\(.*\)\) break;|more = mbar_wait_item_warp\(.*\) && ", line), line
    # the answer of the launch control is read only where it has arrived
    assert re.findall(r"^.*clc_answer\(.*$", text, re.M) == re.findall(r"^.*mbar_wait_item_warp\(&clc_full.*&& clc_answer\(.*$",
                                                                      text, re.M) != []
