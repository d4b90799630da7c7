"""Builds libnvllm_b200_attn.so in-tree with nvcc for sm_100a (cross-compiles without a GPU), and the extension module
that binds it to torch (torch_binding.cpp, host code only).

Usage:  python -m nanovllm_jax_b200.csrc.build [--force] [--verbose]
Each .cu file is compiled to an object next to it and the objects are linked into
``nanovllm_jax_b200/libnvllm_b200_attn.so``.  A file is rebuilt only when it, or a header,
is newer than its object.  The extension is ``nanovllm_jax_b200/_torch_binding.<abi>.so``.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(HERE)
ROOT = os.path.dirname(PKG)
LIB = os.path.join(PKG, "libnvllm_b200_attn.so")
BINDING_SOURCE = os.path.join(HERE, "torch_binding.cpp")
BINDING = os.path.join(PKG, "_torch_binding" + sysconfig.get_config_var("EXT_SUFFIX"))

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def sources() -> list[str]:
    return sorted(os.path.join(HERE, f) for f in os.listdir(HERE) if f.endswith(".cu"))


def _headers_mtime() -> float:
    hs = [os.path.join(HERE, f) for f in os.listdir(HERE) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(ROOT, "include", "nvllm_b200_attn.h"))
    return max(os.path.getmtime(h) for h in hs)


def build_binding(nvcc: str, force: bool = False, verbose: bool = False) -> str:
    header = os.path.join(ROOT, "include", "nvllm_b200_attn.h")
    if not force and os.path.exists(BINDING) and os.path.getmtime(BINDING) >= max(map(os.path.getmtime,
                                                                                     (BINDING_SOURCE, header))):
        return BINDING
    import torch
    root = os.path.dirname(os.path.abspath(torch.__file__))
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    includes = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cmd = [os.environ.get("CXX") or shutil.which("g++") or "c++", "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(f"-isystem{d}" for d in includes), BINDING_SOURCE, "-o", BINDING, "-L" + os.path.join(root, "lib"),
           "-ltorch_python", "-ltorch_cpu", "-lc10_cuda", "-lc10"]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    return BINDING


def build(force: bool = False, verbose: bool = False) -> str:
    nvcc = _nvcc()
    hdr_m = _headers_mtime()
    objs, rebuilt = [], False
    for src in sources():
        obj = src[:-3] + ".o"
        objs.append(obj)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_m):
            cmd = [nvcc, *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-c", src, "-o", obj]
            if verbose:
                print(" ".join(cmd), flush=True)
            subprocess.run(cmd, check=True)
            rebuilt = True
    if rebuilt or not os.path.exists(LIB):
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-cudart", "static"]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.run(cmd, check=True)
    build_binding(nvcc, force, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
