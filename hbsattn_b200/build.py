"""Builds libhbsattn_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU).

    python hbsattn_b200/build.py [--force] [--verbose] [--strict]
    (run as a script: importing the package needs the library)

Beside the C ABI library it builds _host.so, the CPython extension of csrc/hbsa_host.cpp that the Python operators call into
(g++ against the headers and libraries of the torch that is installed; no device code).

--strict also builds libhbsattn_b200_strict.so: the same sources with -DHBSA_STRICT_TCGEN05, in which the MMA
thread of the tensor-core kernel fences after every barrier it observes and waits for the P V products of a lane
to complete before the next S product overwrites their operand.  It exists to check, bit for bit, the ordering
the shipped library relies on (tests/test_gpu_strict_order.py); select it with HBSATTN_B200_LIBRARY=<path>.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libhbsattn_b200.so")
HOST_PATH = os.path.join(PKG_DIR, "_host.so")
HOST_SOURCE = os.path.join(CSRC, "hbsa_host.cpp")
STRICT_LIB_PATH = os.path.join(PKG_DIR, "libhbsattn_b200_strict.so")
SOURCES = ["hbsa_api.cu", "hbsa_schedule.cu", "hbsa_fwd_generic.cu", "hbsa_fwd_sm100.cu",
           "hbsa_bwd_sm100.cu", "hbsa_bwd_generic.cu", "hbsa_static_scratch.cu"]
HEADERS = ["hbsa_common.cuh", "sm100_ptx.cuh", "sm100_common.cuh", os.path.join("..", "..", "include", "hbsattn_b200.h")]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; hbsattn_b200 has no CPU fallback and cannot be built without CUDA")
    return cand


def nvcc_flags(verbose: bool = False):
    # No --split-compile: with it nvcc makes another binary each time (two builds of the same backward differed by 17 % in size) and kernel
    # times moved by up to 20 % from build to build.  Without it a build of everything takes about 50 s.
    flags = ["-O3", "--threads", "8", "-std=c++17", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a",
             "-Xcompiler", "-fPIC", "-I", os.path.join(PKG_DIR, "..", "include")]
    if verbose:
        flags += ["-Xptxas", "-v"]
    return flags


def is_stale(path: str = LIB_PATH) -> bool:
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    deps = [os.path.join(CSRC, s) for s in SOURCES + HEADERS] + [os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False, strict: bool = False) -> str:
    """Compile every CUDA source into hbsattn_b200/libhbsattn_b200.so (or, with strict=True, into
    libhbsattn_b200_strict.so with -DHBSA_STRICT_TCGEN05), and the host extension; returns the library's path."""
    build_host(force)
    out = STRICT_LIB_PATH if strict else LIB_PATH
    if not force and not is_stale(out):
        return out
    cmd = [_nvcc(), "-shared", "-o", out] + nvcc_flags(verbose) + (["-DHBSA_STRICT_TCGEN05"] if strict else []) + \
        [os.path.join(CSRC, s) for s in SOURCES]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed building %s (exit %d)" % (os.path.basename(out), res.returncode))
    return out


def host_tag() -> str:
    """What the host extension is tied to beside its sources: the torch and the Python it was compiled against."""
    import torch
    return f"torch {torch.__version__}, {sys.implementation.cache_tag}"


def host_is_stale(path: str = HOST_PATH) -> bool:
    if not os.path.exists(path):
        return True
    deps = [HOST_SOURCE, os.path.join(PKG_DIR, "..", "include", "hbsattn_b200.h"), os.path.abspath(__file__)]
    if any(os.path.getmtime(d) > os.path.getmtime(path) for d in deps):
        return True
    with open(path, "rb") as f:
        return f"[{host_tag()}]".encode() not in f.read()


def build_host(force: bool = False) -> str:
    """Compile csrc/hbsa_host.cpp into hbsattn_b200/_host.so; returns the path."""
    if not force and not host_is_stale():
        return HOST_PATH
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    libs = ["torch_python", "torch", "torch_cpu", "torch_cuda", "c10", "c10_cuda"]
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", HOST_PATH, HOST_SOURCE, f'-DHBSA_HOST_TAG="[{host_tag()}]"',
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cmd += [f"-I{d}" for d in include] + [f"-L{os.path.join(root, 'lib')}"] + [f"-l{n}" for n in libs]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("g++ failed building _host.so (exit %d)" % res.returncode)
    return HOST_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
    if "--strict" in sys.argv:
        print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv, strict=True))
