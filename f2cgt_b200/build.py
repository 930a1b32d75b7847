"""Build ``libf2cgt_b200.so`` (the C-ABI library, include/f2cgt_b200.h) in-tree with plain nvcc, and ``_native.so``
(the CPython module between torch and the library) with the host compiler.

The library has no torch, pybind or Python dependency: it is CUDA C++ compiled for sm_100a only and
linked against the static CUDA runtime.  The module holds no device code.  ``python -m f2cgt_b200.build`` rebuilds what is stale;
``--force`` rebuilds everything; ``--verbose`` prints ptxas resource usage (-Xptxas -v).
"""
import argparse
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(CSRC, "_obj")
LIB = os.path.join(PKG, "libf2cgt_b200.so")
NATIVE_SRC = os.path.join(PKG, "native")
NATIVE = os.path.join(PKG, "_native.so")
HEADER = os.path.join(os.path.dirname(PKG), "include", "f2cgt_b200.h")

NVCC_FLAGS = ["-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _nvcc():
    return os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")


def _deps_mtime():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))] + [HEADER]
    return max(os.path.getmtime(h) for h in hs)


def _run_all(commands, jobs):
    """[(command, name)] in parallel; raises with the compiler's messages, returns [(name, messages)]."""
    def one(pair):
        r = subprocess.run(pair[0], capture_output=True, text=True)
        return r.returncode, pair[1], r.stderr

    with ThreadPoolExecutor(max_workers=jobs) as ex:
        results = list(ex.map(one, commands))
    for rc, name, err in results:
        if rc != 0:
            raise RuntimeError(f"compiling {name} failed:\n{err[-6000:]}")
    return [(name, err) for _, name, err in results]


def build_native(force=False, jobs=8):
    """The torch-facing module; rebuilt when its sources or the C header change."""
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths, library_paths
    srcs = sorted(os.path.join(NATIVE_SRC, f) for f in os.listdir(NATIVE_SRC) if f.endswith(".cpp"))
    dep_t = max(os.path.getmtime(h) for h in [HEADER] + [os.path.join(NATIVE_SRC, f) for f in os.listdir(NATIVE_SRC) if f.endswith(".h")])
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    inc = [f"-I{d}" for d in include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]]
    flags = ["-std=c++17", "-O2", "-fPIC", "-fvisibility=hidden", "-Wno-deprecated-declarations",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    objs, commands = [], []
    for src in srcs:
        obj = os.path.join(OBJ, "native_" + os.path.basename(src)[:-4] + ".o")
        objs.append(obj)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), dep_t):
            commands.append((["g++"] + flags + inc + ["-c", src, "-o", obj], src))
    _run_all(commands, jobs)
    if commands or not os.path.exists(NATIVE):
        libs = [f"-L{d}" for d in library_paths() + [os.path.join(cuda, "lib64"), PKG]]
        link = ["g++", "-shared", "-o", NATIVE] + objs + libs + ["-l:libf2cgt_b200.so", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
                                                                "-ltorch_python", "-ltorch", "-lcudart", "-lcublas", "-Wl,-rpath,$ORIGIN"]
        _run_all([(link, NATIVE)], 1)
    return NATIVE


def build(force=False, verbose=False, jobs=8):
    os.makedirs(OBJ, exist_ok=True)
    dep_t = _deps_mtime()
    units = [(s, os.path.join(OBJ, os.path.basename(s)[:-3] + ".o")) for s in sources()]

    def compile_one(pair):
        src, obj = pair
        if not force and os.path.exists(obj) and os.path.getmtime(obj) >= max(os.path.getmtime(src), dep_t):
            return 0, src, ""
        cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
        p = subprocess.run(cmd, capture_output=True, text=True)
        return p.returncode, src, p.stderr

    with ThreadPoolExecutor(max_workers=jobs) as ex:
        results = list(ex.map(compile_one, units))
    for rc, src, err in results:
        if rc != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{err[-6000:]}")
        if verbose and err:
            print(f"== {os.path.basename(src)}\n{err}")
    objs = [o for _, o in units]
    if force or not os.path.exists(LIB) or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs):
        cmd = [_nvcc(), "-shared", "-o", LIB, "-gencode", "arch=compute_100a,code=sm_100a"] + objs
        p = subprocess.run(cmd, capture_output=True, text=True)
        if p.returncode != 0:
            raise RuntimeError(f"link failed:\n{p.stderr[-4000:]}")
    build_native(force, jobs)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
    sys.exit(0)
