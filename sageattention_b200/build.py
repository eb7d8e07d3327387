"""Build ``libnvfp4_b200.so`` and ``_native.so`` in-tree.

``python -m sageattention_b200.build`` compiles every ``csrc/*.cu`` for sm_100a with nvcc to an object
(in parallel, skipping objects newer than all sources and headers) and links one shared library next
to this file.  No torch headers are involved: the library is a plain C ABI
(``include/nvfp4_b200.h``).  The operators' host path (``csrc/host/native.cpp``, a Python extension on
torch's C++ API) is compiled with the host compiler beside them and linked against that library, again
when torch is another one than it was compiled against.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libnvfp4_b200.so")
NATIVE_SRC = os.path.join(CSRC, "host", "native.cpp")
NATIVE = os.path.join(HERE, "_native.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or add it to PATH")


def _native_commands(nvcc: str):
    """(compile, link) commands of the host path's Python extension."""
    import torch
    base = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    inc = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cxx = os.environ.get("CXX") or shutil.which("g++") or "c++"
    obj = os.path.join(OBJ, "native.o")
    compile_cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_native",
                   f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                   *(f"-I{d}" for d in inc), "-c", NATIVE_SRC, "-o", obj]
    link_cmd = [cxx, "-shared", "-o", NATIVE, obj, f"-L{HERE}", "-l:libnvfp4_b200.so", f"-L{os.path.join(base, 'lib')}",
                "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"]
    return obj, compile_cmd, link_cmd


def _run(cmd, what: str) -> str:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{r.stdout}\n{r.stderr}")
    return r.stderr


def _native_tag(cmd) -> str:
    """What the host path's object depends on besides its sources: torch (its headers, its ABI) and the command."""
    import torch
    return "\n".join([torch.__version__, str(torch.version.git_version), *cmd])


def _native_stale(obj: str, cmd) -> bool:
    """Older than its sources, or compiled against another torch: the stamp beside the object says which."""
    if not os.path.exists(obj) or not os.path.exists(obj + ".tag"):
        return True
    with open(obj + ".tag") as f:
        if f.read() != _native_tag(cmd):
            return True
    return os.path.getmtime(obj) < max(os.path.getmtime(NATIVE_SRC), os.path.getmtime(_headers()[0]))


def _headers():
    out = [os.path.join(os.path.dirname(HERE), "include", "nvfp4_b200.h")]
    for root, _, files in os.walk(CSRC):
        out += [os.path.join(root, f) for f in files if f.endswith((".cuh", ".h"))]
    return out


def build(verbose: bool = False, force: bool = False) -> str:
    nvcc = _nvcc()
    os.makedirs(OBJ, exist_ok=True)
    sources = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    newest_hdr = max(os.path.getmtime(h) for h in _headers())
    jobs = []
    for src in sources:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ, src[:-3] + ".o")
        stale = force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), newest_hdr)
        cmd = [nvcc, *(["-Xptxas=-v"] if verbose else []), *NVCC_FLAGS, "-c", s, "-o", o]
        jobs.append((cmd, s, o, stale))
    native_obj, native_compile, native_link = _native_commands(nvcc)
    native_stale = force or _native_stale(native_obj, native_compile)
    jobs.append((native_compile, NATIVE_SRC, native_obj, native_stale))

    def compile_one(job):
        cmd, s, _, stale = job
        if not stale:
            return None
        log = _run(cmd, f"compiling {s}")
        return log if verbose else None

    with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
        logs = list(ex.map(compile_one, jobs))
    if native_stale:
        with open(native_obj + ".tag", "w") as f:
            f.write(_native_tag(native_compile))
    if verbose:
        for log in logs:
            if log:
                print(log)
    objs = [o for _, _, o, _ in jobs if o != native_obj]
    if force or not os.path.exists(LIB) or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs):
        _run([nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC"],
             "linking " + LIB)
    if force or not os.path.exists(NATIVE) or os.path.getmtime(native_obj) > os.path.getmtime(NATIVE):
        _run(native_link, "linking " + NATIVE)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
