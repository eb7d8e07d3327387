"""Roles in which a whole warp waits and one of its threads acts: no lane may be left behind in a wait, for what that thread
does lets the barrier go on, and the parity that the late lane looks for comes back only with the phase after the next."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sageattention_b200", "csrc")

WAIT = r"\bmbar_(?:wait|wait_all|spin_wait|wait_item)\("
MEET = r"\b__syncwarp\(\)|\b\w+_sync\(0xffffffffu|\bmbar_wait_(?:item_)?warp\("
ACT = r"\b(?:umma_commit|mbar_arrive|mbar_expect_tx|clc_request)\("


def _without_own_waits(text):
    """text without the blocks of the one thread in which it waits by itself."""
    at = 0
    while (i := text.find("if (leader) {", at)) >= 0:
        depth, j = 0, text.index("{", i)
        while True:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
            if depth == 0:
                break
        if re.search(WAIT, text[i:j]):
            text = text[:i] + text[j:]
        else:
            at = j
    return text


@pytest.mark.parametrize("name,roles", [("fwd.cu", 3), ("bwd.cu", 5), ("bwd_fp4.cu", 2), ("decode.cu", 1)])
def test_lanes_meet_between_a_wait_and_an_act(name, roles):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    starts = [m.start() for m in re.finditer(r"const bool leader = elect_one\(\);", text)]
    assert len(starts) == roles
    for i in starts:
        role = _without_own_waits(text[i:re.compile(r"^  \} else|^}", re.M).search(text, i).start()])
        assert "mbar_" in role
        late = None
        for m in re.finditer(f"({WAIT})|({MEET})|({ACT})", role):
            line = role[role.rindex("\n", 0, m.start()) + 1:role.index("\n", m.start())].strip()
            if m.group(1):
                late = line
            elif m.group(2):
                late = None
            else:
                assert late is None, f"{line} behind {late}"
        assert late is None


def test_the_warp_form_converges():
    text = open(os.path.join(CSRC, "common", "sm100.cuh")).read()
    body = text[text.index("mbar_wait_warp("):]
    assert re.search(r"mbar_wait\(.*\);\s*__syncwarp\(\);", body[:body.index("\n}")])
