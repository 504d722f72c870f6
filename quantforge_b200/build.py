"""Builds libquantforge_rt.so (CUDA kernels + C ABI) for sm_100a with nvcc, and _qf_host.<interpreter>.torch-<version>.so
(the native host path of the Python operators, a CPython extension over torch's C++ API) with g++, in-tree.

    python -m quantforge_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU.  The shared libraries land in quantforge_b200/lib/.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libquantforge_rt.so")

SOURCES = ["qf_api.cu", "qf_unpack.cu", "qf_quantize.cu", "qf_gemv.cu", "qf_gemv_slab.cu", "qf_gemm_tcgen05.cu", "qf_stream.cu",
           "qf_slab_chain.cu", "qf_chain_plan.cu", "qf_tensor_map.cu", "qf_comm.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _older(path: str, deps) -> bool:
    return not os.path.exists(path) or any(os.path.getmtime(d) > os.path.getmtime(path) for d in deps)


def _headers() -> list:
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))] + \
        [os.path.join(ROOT, "include", "quantforge_rt.h"), os.path.abspath(__file__)]


def _stale() -> bool:
    return _older(LIB_PATH, _headers() + [os.path.join(CSRC, f) for f in SOURCES])


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        build_host()
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(LIB_DIR, src.replace(".cu", ".o"))
        objs.append(obj)
        if not force and not verbose and not _older(obj, _headers() + [os.path.join(CSRC, src)]):
            continue
        cmd = [_nvcc(), *NVCC_FLAGS, "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-c",
               os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
            print(" ".join(cmd), flush=True)
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, pr in procs:
        out, _ = pr.communicate()
        if pr.returncode != 0 or verbose:
            print(f"--- {src}\n{out}", flush=True)
        failed |= pr.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    link = [_nvcc(), "-shared", "-o", LIB_PATH, *objs, "-gencode", "arch=compute_100a,code=sm_100a",
            "-Xcompiler", "-fPIC", "-lcudart_static", "-ldl", "-lpthread", "-lrt"]
    subprocess.run(link, check=True)
    build_host(force)
    return LIB_PATH


HOST_SRC = os.path.join(CSRC, "qf_host.cpp")


def build_host(force: bool = False) -> str:
    """Builds the native host path for this interpreter and torch (part of build(): it links against libquantforge_rt.so)."""
    from ._lib import HOST_PATH
    if not force and not _older(HOST_PATH, [HOST_SRC, os.path.join(ROOT, "include", "quantforge_rt.h")]):
        return HOST_PATH
    import torch
    from torch.utils import cpp_extension
    includes = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(ROOT, "include"),
                                                os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared",
                    f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                    *[f for i in includes for f in ("-isystem", i)], HOST_SRC, "-o", HOST_PATH,
                    "-L", LIB_DIR, "-lquantforge_rt", "-Wl,-rpath,$ORIGIN",
                    "-L", torch_lib, "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10"],
                   check=True)
    return HOST_PATH


OPT_SRC = os.path.join(HERE, "opt", "quantforge_opt.cpp")
OPT_BIN = os.path.join(HERE, "bin", "quantforge-opt")


def build_opt(force: bool = False) -> str:
    """Builds the re-hosted quantforge-opt driver (plain C++17, no MLIR dependency)."""
    if not force and os.path.exists(OPT_BIN) and os.path.getmtime(OPT_BIN) >= os.path.getmtime(OPT_SRC):
        return OPT_BIN
    os.makedirs(os.path.dirname(OPT_BIN), exist_ok=True)
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-o", OPT_BIN, OPT_SRC], check=True)
    return OPT_BIN


if __name__ == "__main__":
    print(build_opt(force="--force" in sys.argv))
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
