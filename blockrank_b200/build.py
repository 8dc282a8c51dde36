"""Build libblockrank_b200.so (nvcc, sm_100a) and _host.so (g++, the native path from PyTorch tensors to it) in-tree.

    python -m blockrank_b200.build [--force] [--verbose]

libblockrank_b200.so is a plain C-ABI shared object (include/blockrank_b200.h); it is
loaded with ctypes by blockrank_b200._lib.  _host.so is a Python extension module linked against it and against
PyTorch.  Each is rebuilt when any of its sources is newer than the binary.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libblockrank_b200.so")
HOST_LIB = os.path.join(PKG, "_host.so")
HOST_SOURCE = os.path.join(CSRC, "torch_host.cpp")
HEADER = os.path.join(os.path.dirname(PKG), "include", "blockrank_b200.h")
SOURCES = ["brk_api.cu", "attn_simt.cu", "attn_f32.cu", "attn_tc.cu", "attn_bwd.cu", "attn_bwd_mma.cu", "attn_bwd_tc.cu", "attn_bwd_f32.cu",
           "scores.cu",
           "raw_scores.cu", "elementwise.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: libblockrank_b200.so cannot be built")


def sources():
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def needs_build() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = sources() + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    deps.append(HEADER)
    return any(os.path.getmtime(d) > t for d in deps)


def _build_host(verbose: bool) -> subprocess.Popen:
    """Start the compilation of _host.so's object (PyTorch's headers take a minute)."""
    import torch
    from torch.utils.cpp_extension import include_paths
    inc = [*include_paths(), sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include"),
           "/usr/local/cuda/include"]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host",
           "-DTORCH_API_INCLUDE_EXTENSION_H", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           *(f"-I{d}" for d in inc), "-c", HOST_SOURCE, "-o", HOST_SOURCE[:-4] + ".o"]
    if verbose:
        sys.stderr.write(" ".join(cmd) + "\n")
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _link_host(proc: subprocess.Popen) -> None:
    out, _ = proc.communicate()
    if proc.returncode != 0:
        raise RuntimeError("building _host.so failed:\n" + out)
    import torch
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    # libstdc++.so.6 by name: the one that PyTorch has loaded.  A compiler whose own libstdc++ is only there as an archive would
    # link that in, and a second copy of the library in one process does not work: the first number written into an error
    # message went through the wrong locale facet and ended the process.
    link = [os.environ.get("CXX", "g++"), "-shared", "-o", HOST_LIB + ".tmp", HOST_SOURCE[:-4] + ".o", "-l:libstdc++.so.6", LIB,
            f"-L{lib}", "-lc10",
            "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", "-L/usr/local/cuda/lib64", "-lcudart",
            "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{lib}"]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError("linking _host.so failed:\n" + r.stdout)
    os.replace(HOST_LIB + ".tmp", HOST_LIB)


def needs_host_build() -> bool:
    return not os.path.exists(HOST_LIB) or any(os.path.getmtime(d) > os.path.getmtime(HOST_LIB) for d in (HOST_SOURCE, HEADER, os.path.abspath(__file__)))


def build(force: bool = False, verbose: bool = False) -> str:
    host = _build_host(verbose) if force or needs_host_build() else None
    if force or needs_build():
        _build_library(verbose)
    if host is not None:
        _link_host(host)
    return LIB


def _build_library(verbose: bool) -> None:
    objs = []
    procs = []
    for src in sources():
        obj = src[:-3] + ".o"
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- {os.path.basename(src)} ---\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed building libblockrank_b200.so")
    link = [_nvcc(), "-shared", "-Xlinker", "-soname=libblockrank_b200.so", "-o", LIB + ".tmp", *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n" + r.stdout)
    os.replace(LIB + ".tmp", LIB)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
