"""The order of griddepcontrol.wait and .launch_dependents in every kernel, against the rules of
csrc/common/launch.cuh: a late waiter's predecessor must wait before it signals, which no run is sure to show."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sageattention_b200", "csrc")


def _kernels():
    """name -> (file, body) of every __global__ function."""
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s+)?(\w+)\s*\(", text):
            end = re.compile(r"^}", re.M).search(text, m.end()).start()
            out[m.group(1)] = (f, text[m.end():end])
    return out


def _pairs():
    """(late waiter, [predecessors]) as the header lists them."""
    text = open(os.path.join(CSRC, "common", "launch.cuh")).read()
    block = text[text.index("// Late waiters"):text.index("#pragma once")]
    rows = re.findall(r"^//   (\w+)\s+.*?behind ([^(]*)\(", block, re.M)
    return [(k, re.findall(r"\w+_kernel", before)) for k, before in rows]


def test_late_waiters_and_their_predecessors():
    kernels = _kernels()
    late = {n for n, (_, body) in kernels.items() if "late_wait" in body}
    pairs = _pairs()
    assert late == {k for k, _ in pairs}, "the header's list and the kernels that wait late disagree"
    for k, before in pairs:
        body = kernels[k][1]
        assert len(re.findall(r"^  griddep_start\(p\.late_wait != 0[,)]", body, re.M)) == 1
        # the wait at the end, behind which no thread touches operands any more
        tail = body[body.index("if (p.late_wait) griddep_wait();"):]
        assert "tma_" not in tail and "mbar_" not in tail
        assert before
        for n in before:
            b = kernels[n][1]
            wait = re.search(r"griddep_(wait\(\);|start\(p\.late_wait != 0)", b).start()
            assert wait < b.index("griddep_launch();"), f"{n} signals before it waits"


def test_every_other_kernel_waits_unconditionally():
    kernels = _kernels()
    late = {k for k, _ in _pairs()}
    with_pdl = {n for n, (_, b) in kernels.items() if "griddep_" in b}
    assert len(with_pdl) >= 20
    for n in with_pdl - late:
        assert re.search(r"^  griddep_wait\(\);", kernels[n][1], re.M), n
    for f in {kernels[n][0] for n in with_pdl}:      # ... and all of them are launched with the attribute
        assert "<<<" not in open(os.path.join(CSRC, f)).read(), f
    assert {kernels[n][0] for n in kernels if n not in with_pdl} == {"peak.cu", "selftest.cu"}
