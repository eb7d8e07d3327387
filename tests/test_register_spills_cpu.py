"""Kernels that were built to keep within their registers do: no spilled bytes in what the assembler reports."""

import os
import re
import shutil
import subprocess

import pytest

from sageattention_b200 import build as B

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def _spilled(source, tmp_path):
    """kernel -> (bytes stored, bytes loaded)"""
    r = subprocess.run([NVCC, *B.NVCC_FLAGS, "-Xptxas", "-v", "-c", os.path.join(B.CSRC, source), "-o", str(tmp_path / "o.o")],
                       capture_output=True, text=True, check=True)
    found = re.findall(r"Compiling entry function '(\S+)'.*?(\d+) bytes spill stores, (\d+) bytes spill loads", r.stderr, re.S)
    return {k: (int(a), int(b)) for k, a, b in found}


@pytest.mark.parametrize("source,part,kernels", [("vproj.cu", "vproj_pack_kernel", 8),
                                                 ("bwd.cu", "bwd_dkdv_kernelILi256E.*Lb1E", 3)])
def test_no_spills(source, part, kernels, tmp_path):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    spilled = {k: v for k, v in _spilled(source, tmp_path).items() if re.search(part, k)}
    assert len(spilled) == kernels
    assert {k: v for k, v in spilled.items() if v != (0, 0)} == {}
