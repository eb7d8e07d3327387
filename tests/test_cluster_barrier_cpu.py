"""Cluster barriers are `.aligned`: the lanes of a warp have to arrive together, which code with per-lane branches and loops
in front of the barrier does not see to by itself."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sageattention_b200", "csrc")


def test_warps_converge_in_front_of_a_cluster_barrier():
    barriers = 0
    for root, _, files in os.walk(CSRC):
        for name in files:
            if not name.endswith((".cu", ".cuh")):
                continue
            text = re.sub(r"//[^\n]*", "", open(os.path.join(root, name)).read())
            for m in re.finditer(r"barrier\.cluster\.arrive[\w.:]*\.aligned", text):
                statement = text.rindex("asm volatile", 0, m.start())
                assert text[:statement].rstrip().endswith("__syncwarp();"), name
                barriers += 1
    assert barriers >= 1
