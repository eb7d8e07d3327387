"""What kernels do when a wait has run out: a hand-over of work items (csrc/fwd.cu, csrc/bwd.cu) that did not come is never
taken for an item, and a CTA lets its copies land before its memory is another's."""

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


def test_every_kernel_with_waits_reports_and_drains_before_it_gives_up_its_memory():
    seen = 0
    for name in sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__shared__ int err\b", text):
            body = text[m.start():re.compile(r"^}", re.M).search(text, m.start()).start()]
            tail = body[body.rindex("__syncthreads();"):]
            assert re.search(r"report_error(_call)?\(&err, ", tail), name
            assert "tmem_dealloc" not in body or tail.index("report_error") < tail.index("tmem_dealloc"), name
            seen += 1
    assert seen == 8
