"""Roles in which a whole warp waits and one of its threads acts: no lane may be left behind in a wait, for what that thread
issues lets the barrier go on, and the parity that the late lane looks for comes back only with the phase after the next."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sageattention_b200", "csrc")


def _without_blocks(text, head):
    """text without the braced blocks that `head` opens."""
    while (i := text.find(head)) >= 0:
        depth, j = 0, text.index("{", i)
        while True:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
            if depth == 0:
                break
        text = text[:i] + text[j:]
    return text


@pytest.mark.parametrize("name,roles", [("fwd.cu", 3), ("bwd.cu", 5), ("bwd_fp4.cu", 2), ("decode.cu", 1)])
def test_lanes_leave_a_wait_together(name, roles):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    starts = [m.start() for m in re.finditer(r"const bool leader = elect_one\(\);", text)]
    assert len(starts) == roles
    for i in starts:
        role = text[i:re.compile(r"^  \} else|^}", re.M).search(text, i).start()]
        role = _without_blocks(role, "if (leader) {")            # waits of the one thread
        assert "mbar_" in role
        alone = re.findall(r"\bmbar_(?:wait|wait_all|spin_wait|wait_item)\(.*", role)
        assert alone == [], alone


def test_the_warp_forms_converge():
    text = open(os.path.join(CSRC, "common", "sm100.cuh")).read()
    for f in ("mbar_wait_warp", "mbar_wait_all_warp"):
        body = text[text.index(f + "("):]
        body = body[:body.index("\n}")]
        assert re.search(r"mbar_wait(_all)?\(.*\);\s*__syncwarp\(\);", body), f
