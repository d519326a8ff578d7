"""Builds libetcuda.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

    python -m effect_torch_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU. The library sits next to this file so it travels with the
source tree; nothing is installed into site-packages.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libetcuda.so")
CALLS = os.path.join(HERE, "_calls" + sysconfig.get_config_var("EXT_SUFFIX"))  # the extension module of calls.cpp, for this interpreter
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]


def _nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA backend cannot be built")


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cpp")))


def _stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh"))
    deps.append(os.path.join(os.path.dirname(HERE), "include", "et_cuda.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build_calls(force: bool = False) -> None:
    """The CPython module that calls the library without ctypes. Without the interpreter's headers, or where it does not
    compile, there is none (_ThroughCtypes stands in): no module of an older header stays, and none that any interpreter loads."""
    src, header = os.path.join(HERE, "calls.cpp"), os.path.join(os.path.dirname(HERE), "include", "et_cuda.h")
    newest = max(map(os.path.getmtime, (src, header)))
    for module in glob.glob(os.path.join(HERE, "_calls*.so")):
        if os.path.basename(module) == "_calls.so" or os.path.getmtime(module) <= newest or (force and module == CALLS):
            os.remove(module)
    include = sysconfig.get_paths()["include"]
    if os.path.exists(CALLS) or not os.path.exists(os.path.join(include, "Python.h")):
        return
    host_cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    command = [host_cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-I", include, src, "-o", CALLS, "-L", HERE,
               "-l:" + os.path.basename(LIB), "-Wl,-rpath,$ORIGIN"]
    try:
        subprocess.run(command, check=True, stderr=subprocess.PIPE, text=True)
    except (OSError, subprocess.CalledProcessError) as error:
        sys.stderr.write(f"--- calls.cpp: no extension module, its operators go through ctypes\n{getattr(error, 'stderr', None) or error}\n")


def build(force: bool = False, verbose: bool = False) -> str:
    if force or _stale():
        _build_library(verbose)
    build_calls(force)
    return LIB


def _build_library(verbose: bool) -> None:
    objs = []
    build_dir = os.path.join(HERE, "build")
    os.makedirs(build_dir, exist_ok=True)
    host_cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    common = ["-ccbin", host_cxx, "-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC,-fvisibility=hidden",
              "--expt-relaxed-constexpr"] + ARCH_FLAGS
    if verbose:
        common += ["-Xptxas", "-v"]
    procs = []
    for src in sources():
        obj = os.path.join(build_dir, os.path.basename(src) + ".o")
        objs.append(obj)
        extra = ["-x", "cu"] if src.endswith(".cpp") else []
        cmd = [_nvcc()] + common + extra + ["-c", src, "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- {os.path.basename(src)}\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed (see output above)")
    link = [_nvcc(), "-ccbin", host_cxx, "-shared", "-o", LIB] + objs + ["-lcudart"] + ARCH_FLAGS
    subprocess.run(link, check=True)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
