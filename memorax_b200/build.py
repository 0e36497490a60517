"""Builds ``libmxk.so`` (the C-ABI library with every CUDA kernel) in-tree with
nvcc for sm_100a, and ``_C.so`` (the native host code) over it.  ``python -m memorax_b200.build`` or ``build_library()``."""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG_DIR)
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(ROOT, "include")
LIB_PATH = os.path.join(PKG_DIR, "libmxk.so")
OBJ_DIR = os.path.join(PKG_DIR, "build")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-I", INCLUDE, "-I", CSRC,
]


BIND = os.path.join(CSRC, "bind")
BIND_PATH = os.path.join(PKG_DIR, "_C.so")


def _nvcc():
    cand = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"
    return cand if os.path.exists(cand) else "nvcc"


def _sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return hs


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_library(force: bool = False, verbose: bool = False, extra_flags=()) -> str:
    """Compile every ``csrc/*.cu`` for sm_100a and link ``libmxk.so`` next to
    this file.  Rebuilds only what is older than its sources."""
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = _headers()
    jobs = []
    objs = []
    for src in _sources():
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [_nvcc(), *NVCC_FLAGS, *extra_flags, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("build failed: %s\n%s\n%s" % (" ".join(cmd), res.stdout, res.stderr))
        return res.stderr

    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as pool:
            for log in pool.map(run, jobs):
                if verbose and log:
                    sys.stderr.write(log)
    if force or jobs or _stale(LIB_PATH, objs):
        run([_nvcc(), "-shared", "-o", LIB_PATH, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcuda"])
    _build_binding(force, run)
    return LIB_PATH


def _build_binding(force, run):
    """``_C.so``: the native host code over ``libmxk.so`` (g++ against torch's headers)."""
    from torch.utils import cpp_extension
    import sysconfig
    import torch
    sources = sorted(os.path.join(BIND, f) for f in os.listdir(BIND) if f.endswith(".cpp"))
    headers = _headers() + [os.path.join(BIND, f) for f in os.listdir(BIND) if f.endswith(".h")]
    include = [*cpp_extension.include_paths("cuda"), sysconfig.get_paths()["include"], INCLUDE, CSRC]
    flags = ["-O2", "-std=c++17", "-fPIC", "-DTORCH_EXTENSION_NAME=_C", "-DTORCH_API_INCLUDE_EXTENSION_H",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(x for i in include for x in ("-isystem", i))]
    objs = [os.path.join(OBJ_DIR, "bind_" + os.path.basename(src)[:-4] + ".o") for src in sources]
    jobs = [["g++", *flags, "-c", src, "-o", obj] for src, obj in zip(sources, objs) if force or _stale(obj, [src] + headers)]
    with ThreadPoolExecutor(max_workers=max(1, min(8, len(jobs)))) as pool:
        list(pool.map(run, jobs))
    if force or jobs or _stale(BIND_PATH, objs + [LIB_PATH]):
        torch_lib = cpp_extension.library_paths("cuda")[0]
        run(["g++", "-shared", "-o", BIND_PATH, *objs, "-L", PKG_DIR, "-l:libmxk.so", "-Wl,-rpath,$ORIGIN", "-L", torch_lib,
             "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda"])


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
