"""Compile the CUDA sources into cula_b200/lib/libcula_kda.so for sm_100a with nvcc, and the native host path (argument
checks, allocation, autograd, launches; C++ on libtorch) into the Python extension cula_b200/lib/_host.so with g++.

    python -m cula_b200.build [--force] [--verbose]

The library is built in-tree and loaded with ctypes (cula_b200/_native.py); it has a plain C ABI
(include/cula_kda.h) and links only against the CUDA runtime (the one driver function it needs, the tensor-map encoder
of the stages that move data by TMA, is looked up through the runtime's driver entry point at first use).
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB = os.path.join(LIB_DIR, "libcula_kda.so")
OBJ_DIR = os.path.join(PKG, "build")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _deps_mtime():
    files = glob.glob(os.path.join(CSRC, "*")) + glob.glob(os.path.join(PKG, "..", "include", "*.h"))
    return max(os.path.getmtime(f) for f in files)


HOST_SRC = os.path.join(CSRC, "host")
HOST_LIB = os.path.join(LIB_DIR, "_host.so")


def build_host(force=False):
    """Build cula_b200/lib/_host.so. It reaches the kernels through the C ABI of libcula_kda.so, which it loads at run time."""
    deps = glob.glob(os.path.join(HOST_SRC, "*")) + [os.path.join(PKG, "..", "include", "cula_kda.h")]
    if not force and os.path.exists(HOST_LIB) and os.path.getmtime(HOST_LIB) >= max(os.path.getmtime(f) for f in deps):
        return HOST_LIB
    import torch
    from torch.utils import cpp_extension
    os.makedirs(OBJ_DIR, exist_ok=True)
    os.makedirs(LIB_DIR, exist_ok=True)
    cuda_home = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    includes = [*cpp_extension.include_paths(), os.path.join(cuda_home, "include"), sysconfig.get_paths()["include"]]
    flags = ["-O2", "-std=c++17", "-fPIC", "-DTORCH_EXTENSION_NAME=_host", "-DTORCH_API_INCLUDE_EXTENSION_H",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{i}" for i in includes)]
    procs = []
    for src in sorted(glob.glob(os.path.join(HOST_SRC, "*.cpp"))):
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-4] + ".host.o")
        procs.append((obj, subprocess.Popen([os.environ.get("CXX", "g++"), *flags, "-c", src, "-o", obj])))
    if any(p.wait() != 0 for _, p in procs):
        raise RuntimeError("g++ failed")
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    subprocess.run([os.environ.get("CXX", "g++"), "-shared", "-o", HOST_LIB, *(o for o, _ in procs), f"-L{torch_lib}", f"-L{cuda_home}/lib64",
                    "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch_python", "-lcudart", "-ldl"], check=True)
    return HOST_LIB


TIMERS_LIB = os.path.join(LIB_DIR, "libcula_kda_timers.so")


def build(force=False, verbose=False, timers=False):
    """Build the library. ``timers=True`` builds a second library, libcula_kda_timers.so, with -DKDA_PHASE_TIMERS:
    the chunk-parallel forward kernel and the gated backward kernel then count clock64() cycles per phase (see
    cula_b200/phase_timers.py); it is a profiling aid and is never loaded by the package itself."""
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    os.makedirs(LIB_DIR, exist_ok=True)
    obj_dir = OBJ_DIR + ("_timers" if timers else "")
    lib = TIMERS_LIB if timers else LIB
    os.makedirs(obj_dir, exist_ok=True)
    if not force and os.path.exists(lib) and os.path.getmtime(lib) >= _deps_mtime():
        return lib
    extra = (["-Xptxas", "-v"] if verbose else []) + (["-DKDA_PHASE_TIMERS"] if timers else [])
    procs, objs = [], []
    for src in sources():
        obj = os.path.join(obj_dir, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        procs.append((src, subprocess.Popen([nvcc, *NVCC_FLAGS, *extra, "-c", src, "-o", obj],
                                            stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, pr in procs:
        out, _ = pr.communicate()
        if pr.returncode != 0 or verbose:
            sys.stderr.write(f"--- {os.path.basename(src)} ---\n{out}\n")
        failed |= pr.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    subprocess.run([nvcc, "-shared", "-o", lib, *objs, "-lcudart"], check=True)
    return lib


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv, timers="--timers" in sys.argv))
    print(build_host(force="--force" in sys.argv))
