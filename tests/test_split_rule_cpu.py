"""The rule that splits a key tile's steps over a cluster, at sizes where the times of every split are known."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SOURCE = r"""
#include "common/bwd_util.cuh"
#include <cstdio>
int main() {
  const int slots[4] = {148, 74, 33, 15};
  long long tiles, longest, shortest;
  int packed;
  while (scanf("%lld %lld %lld %d", &tiles, &longest, &shortest, &packed) == 4)
    printf("%d\n", nvfp4::cluster_split(tiles, longest, shortest, packed != 0, slots));
}
"""

# (key heads, query heads, tokens, D, block-scaled, samples) -> microseconds of the backward with 1, 2, 4 and 8 CTAs a tile
MEASURED = {
    (8, 8, 256, 128, False, 0): (15.3, 15.7, 15.5, 29.0),
    (4, 16, 1024, 128, False, 0): (67.9, 44.6, 36.8, 56.2),
    (2, 8, 2048, 128, False, 0): (121.5, 73.5, 50.0, 75.1),
    (8, 32, 256, 128, False, 0): (26.1, 21.6, 18.9, 29.4),
    (8, 32, 1024, 128, False, 0): (84.1, 58.9, 67.6, 97.4),
    (4, 16, 8192, 128, False, 0): (770.2, 887.0, 943.4, 1094.1),
    (8, 8, 256, 256, True, 0): (34.0, 34.5, 35.8, 64.7),
    (4, 16, 1024, 256, True, 0): (127.6, 94.4, 94.2, 129.8),
    (2, 8, 2048, 128, True, 0): (177.9, 114.0, 83.3, 107.9),
    (2, 8, 8192, 256, True, 0): (1106.8, 731.6, 865.0, 1024.3),
    (2, 8, 8192, 128, False, 4): (317.8, 208.3, 218.4, 288.9),
    (4, 16, 4096, 128, True, 2): (362.7, 228.5, 270.1, 345.9),
}


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cu").write_text(SOURCE)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(ROOT, "sageattention_b200", "csrc"), "-o", str(d / "rule"), str(d / "rule.cu")], check=True)

    def ask(cases):
        text = "\n".join(" ".join(map(str, c)) for c in cases)
        out = subprocess.run([str(d / "rule")], input=text, capture_output=True, text=True, check=True).stdout
        return [int(x) for x in out.split()]
    return ask


def test_split_is_near_the_best_measured_one(rule):
    cases = []
    for hk, h, s, d, scaled, samples in MEASURED:
        g, unit = h // hk, 128 if scaled else 64
        tiles = hk * -(-s // 128) * (1 if scaled else d // 128)
        cases.append((tiles, g * -(-s // unit), g if scaled else 2 * g, int(samples > 0)))
    for key, n in zip(MEASURED, rule(cases)):
        times = MEASURED[key]
        assert times[n.bit_length() - 1] <= 1.16 * min(times), (key, n, times)


def test_split_fits_the_steps_of_few_and_of_many_tiles(rule):
    assert rule([(1, 1, 1, 0)]) == [1]                # nothing to share
    assert rule([(1, 4096, 4096, 0)]) == [8]          # one long tile
    assert rule([(15, 4096, 4096, 0)]) == [8]         # as many as clusters of eight are resident
    assert rule([(16, 4096, 4096, 0)]) == [4]         # one more would be a second wave
    assert rule([(10 ** 6, 4096, 2, 0)]) == [1]
