"""The C side keeps nothing between calls but texts and plans: in particular nothing by the address of an operand."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sageattention_b200", "csrc")


def test_state_of_a_thread_is_the_error_text_and_the_decode_plan():
    found = []
    for root, _, files in os.walk(CSRC):
        for f in sorted(files):
            text = re.sub(r"//[^\n]*", "", open(os.path.join(root, f)).read())
            found += [(f, line.strip()) for line in text.splitlines() if "thread_local" in line]
    assert sorted(f for f, _ in found) == ["abi.cu", "decode.cu"], found
    text = open(os.path.join(CSRC, "decode.cu")).read()
    memo = re.search(r"struct Memo \{([^}]*)\}", text).group(1)
    assert "*" not in memo and "uintptr_t" not in memo           # sizes only: a plan is a function of them
