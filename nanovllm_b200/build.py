"""Builds the two compiled parts of the package in-tree:

    python -m nanovllm_b200.build [--force] [--verbose]

* libb200attn.so -- the C-ABI CUDA library (include/b200_attn.h), nvcc for sm_100a.  It links the CUDA runtime
  statically and resolves the one driver entry point it needs at run time, so the build needs no GPU and the result
  loads on a machine without a driver.
* _native.<abi>.so -- the Python binding of its hot entry points (csrc/native.cpp), g++ against the installed torch;
  it links the library above by name (found next to it).
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
HEADER = os.path.join(os.path.dirname(PKG_DIR), "include", "b200_attn.h")
LIB_PATH = os.path.join(PKG_DIR, "libb200attn.so")
NATIVE_SOURCE = os.path.join(CSRC, "native.cpp")
NATIVE_PATH = os.path.join(PKG_DIR, "_native" + sysconfig.get_config_var("EXT_SUFFIX"))
SOURCES = ["host.cu", "store_kvcache.cu", "decode_attn.cu", "decode_cluster.cu", "prefill_attn_mma.cu", "prefill_attn_tc2.cu", "prefill_attn.cu", "qk_norm_rope_store.cu", "decode_metadata.cu", "small_allreduce.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-shared", "-Xcompiler", "-fPIC"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: cannot build libb200attn.so (set NVCC=/path/to/nvcc)")


def _older(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def _run(cmd, what, verbose):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError("building %s failed (exit %d)" % (what, res.returncode))


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles the C-ABI library if it is missing or older than its sources; returns its path."""
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".cpp")] + [HEADER]
    if force or _older(LIB_PATH, deps):
        _run([_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB_PATH] +
             [os.path.join(CSRC, s) for s in SOURCES], "libb200attn.so", verbose)
    return LIB_PATH


def build_native(force: bool = False, verbose: bool = False) -> str:
    """The same for the Python binding (and the library it links); returns its path."""
    build(force, verbose)
    if force or _older(NATIVE_PATH, [NATIVE_SOURCE, HEADER]):
        import torch
        from torch.utils.cpp_extension import include_paths, library_paths
        cuda_home = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
        cmd = [os.environ.get("CXX") or shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC",
               "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)]
        for inc in include_paths() + [os.path.join(cuda_home, "include"), sysconfig.get_paths()["include"]]:
            cmd += ["-isystem", inc]
        cmd += ["-o", NATIVE_PATH, NATIVE_SOURCE]
        for lib in library_paths():
            cmd += ["-L" + lib]
        # the CUDA runtime is torch's own (already loaded with it)
        cmd += ["-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10", "-L" + PKG_DIR,
                "-lb200attn", "-Wl,-rpath,$ORIGIN", "-Wl,--allow-shlib-undefined"]
        _run(cmd, os.path.basename(NATIVE_PATH), verbose)
    return NATIVE_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
    print(build_native(verbose="--verbose" in sys.argv))
