"""Resident clusters are remembered by size only for kernels of which an SM holds one block; a size that no cluster has is
refused.  The runtime's answers are made up here."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SOURCE = r"""
#include <cuda_runtime.h>
#include <cstdio>
static int asked = 0;
static cudaError_t fake_device(int* dev) { *dev = 0; return cudaSuccess; }
static cudaError_t fake_clusters(int* n, const void*, const cudaLaunchConfig_t* c) {
  ++asked;
  *n = 148 * (int)(228 * 1024 / (c->dynamicSmemBytes + 1024)) / (int)c->attrs[0].val.clusterDim.z;
  return cudaSuccess;
}
#define cudaGetDevice fake_device
#define cudaOccupancyMaxActiveClusters fake_clusters
#include "common/launch.cuh"
char* nvfp4::last_error_buffer() { static char text[512]; return text; }
static char a, b, c;
int main() {
  using nvfp4::cluster_slots;
  const int big = 200 * 1024, other = 150 * 1024, small = 50 * 1024;
  printf("%d ", cluster_slots(&a, 384, small, 148, 2));      // four blocks an SM
  printf("%d ", cluster_slots(&b, 384, big, 148, 2));
  printf("%d ", cluster_slots(&c, 256, other, 148, 2));
  printf("%d ", cluster_slots(&a, 384, small, 148, 2));
  printf("%d ", asked);
  printf("%d %d %d\n", cluster_slots(&b, 384, big, 148, 0), cluster_slots(&b, 384, big, 148, 9), cluster_slots(&b, 384, big, 148, -1));
}
"""


def test_answers_are_kept_where_they_depend_on_the_size_alone(tmp_path):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    (tmp_path / "slots.cu").write_text(SOURCE)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(ROOT, "sageattention_b200", "csrc"), "-o", str(tmp_path / "slots"), str(tmp_path / "slots.cu")],
                   check=True)
    out = subprocess.run([str(tmp_path / "slots")], capture_output=True, text=True, check=True).stdout.split()
    # the small kernel is asked for every time, the second of the two large ones is not
    assert [int(x) for x in out] == [296, 74, 74, 296, 3, 0, 0, 0]
