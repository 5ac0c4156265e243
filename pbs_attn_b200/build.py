"""Builds libpbs_b200.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

    python -m pbs_attn_b200.build [--force] [--verbose]

Beside it pbs_host.so, the native host side of the Python call (csrc/host_call.cpp, against the installed torch).
Objects and the libraries land in pbs_attn_b200/lib/ (git-ignored).  nvcc cross-compiles
without a GPU.  The library links the static CUDA runtime only, so it also loads on a
machine without a driver (the symbol-export test does that).
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "lib")
LIB = os.path.join(OUT, "libpbs_b200.so")
HOST_SRC, HOST = os.path.join(CSRC, "host_call.cpp"), os.path.join(OUT, "pbs_host.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I", INCLUDE,
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _host_command():
    import torch
    from torch.utils import cpp_extension
    import sysconfig
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    includes = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    libdir = os.path.join(os.path.dirname(torch.__file__), "lib")
    return (["g++", "-O2", "-shared", "-fPIC", "-std=c++17", "-Wno-attributes", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
            + [f for d in includes for f in ("-isystem", d)] + [HOST_SRC, "-o", HOST, "-L" + libdir, "-L" + os.path.join(cuda, "lib64"),
               "-ltorch_python", "-ltorch_cpu", "-lc10_cuda", "-lc10", "-l:libcudart.so.12"])


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OUT, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(INCLUDE, "pbs_b200.h"))
    nvcc = _nvcc()
    jobs = []
    objs = []
    for src in sources():
        obj = os.path.join(OUT, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed: " + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    objects = len(jobs)
    if force or _stale(HOST, [HOST_SRC, os.path.join(INCLUDE, "pbs_b200.h")]):
        jobs.append(_host_command())
    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for log in ex.map(run, jobs):
            if verbose and log:
                print(log)
    if force or objects or _stale(LIB, objs):
        run([nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB] + objs)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
