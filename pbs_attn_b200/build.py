"""Builds libpbs_b200.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

    python -m pbs_attn_b200.build [--force] [--verbose]

Beside it pbs_host.<torch>.<python>.so, the native host side of the Python call (csrc/host_call.cpp), which fits the torch and Python
in its name alone.  Where it could not be built or was built for others calls go through Python.
Objects and the libraries land in pbs_attn_b200/lib/ (git-ignored).  nvcc cross-compiles
without a GPU.  The library links the static CUDA runtime only, so it also loads on a
machine without a driver (the symbol-export test does that).
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
OUT = os.path.join(HERE, "lib")
LIB = os.path.join(OUT, "libpbs_b200.so")
HOST_SRC = os.path.join(CSRC, "host_call.cpp")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I", INCLUDE,
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        path = cand and shutil.which(cand)
        if path:
            return path
    raise RuntimeError("nvcc not found")


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def host_path() -> str:
    """pbs_host for the installed torch and this Python."""
    import torch
    return os.path.join(OUT, f"pbs_host.torch-{torch.__version__}.{sysconfig.get_config_var('SOABI')}.so")


def _host_command(target: str):
    import torch
    from torch.utils import cpp_extension
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    includes = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    libdir = os.path.join(os.path.dirname(torch.__file__), "lib")
    return (["g++", "-O2", "-shared", "-fPIC", "-std=c++17", "-Wno-attributes", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
            + [f for d in includes for f in ("-isystem", d)] + [HOST_SRC, "-o", target, "-L" + libdir, "-L" + os.path.join(cuda, "lib64"),
               "-ltorch_python", "-ltorch_cpu", "-lc10_cuda", "-lc10", f"-l:libcudart.so.{torch.version.cuda.split('.')[0]}"])


def _build_host(run, force: bool):
    try:
        target = host_path()
        if force or _stale(target, [HOST_SRC, os.path.join(INCLUDE, "pbs_b200.h")]):
            for f in os.listdir(OUT):
                if f.startswith("pbs_host."):
                    os.remove(os.path.join(OUT, f))        # for another torch or Python
            run(_host_command(target))
    except Exception as e:                                 # no torch, headers or compiler here: the library needs none of them
        print(f"pbs_host was not built, calls will go through Python: {e}", file=sys.stderr)


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
            raise RuntimeError("failed: " + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    with ThreadPoolExecutor(max_workers=min(8, len(jobs) + 1)) as ex:
        beside = ex.submit(_build_host, run, force)
        for log in ex.map(run, jobs):
            if verbose and log:
                print(log)
        if force or jobs or _stale(LIB, objs):
            run([nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB] + objs)
        beside.result()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
