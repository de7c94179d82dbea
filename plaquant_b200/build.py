"""Builds libplq_b200.so (the C-ABI CUDA library, nvcc for sm_100a) and _plq_torch.so (its PyTorch front end, host
compiler) in-tree.

    python -m plaquant_b200.build            # build what is older than its sources
    python -m plaquant_b200.build --force
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_PATH = os.path.join(HERE, "libplq_b200.so")
SOURCES = ["plq_api.cu", "plq_pack.cu", "plq_gemv.cu", "plq_gemv_tc.cu", "plq_gemm.cu", "plq_gptq.cu", "plq_rope.cu"]
HEADERS = ["plq_common.cuh", "plq_quant.cuh", "plq_tc.cuh", os.path.join("..", "..", "include", "plq.h")]
TORCH_LIB_PATH = os.path.join(HERE, "_plq_torch.so")
TORCH_SOURCES = ["plq_torch.cpp", os.path.join("..", "..", "include", "plq.h")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--shared",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or add it to PATH")


def needs_build() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    return any(os.path.getmtime(os.path.join(CSRC, f)) > t for f in SOURCES + HEADERS)


def build_library(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB_PATH
    cmd = [_nvcc(), *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []),
           *[os.path.join(CSRC, f) for f in SOURCES], "-o", LIB_PATH]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stderr)
    return LIB_PATH


def build_torch_front_end(force: bool = False) -> str:
    t = os.path.getmtime(TORCH_LIB_PATH) if os.path.exists(TORCH_LIB_PATH) else -1.0
    if not force and all(os.path.getmtime(os.path.join(CSRC, f)) <= t for f in TORCH_SOURCES):
        return TORCH_LIB_PATH
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-DTORCH_EXTENSION_NAME=_plq_torch",
           *[f"-I{d}" for d in inc], os.path.join(CSRC, TORCH_SOURCES[0]), "-o", TORCH_LIB_PATH, f"-L{os.path.join(root, 'lib')}", "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_python", "-ldl"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed:\n" + res.stdout + res.stderr)
    return TORCH_LIB_PATH


if __name__ == "__main__":
    build_library(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(LIB_PATH, build_torch_front_end(force="--force" in sys.argv))
