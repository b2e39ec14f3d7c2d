"""Builds libqk_cuda.so in-tree with nvcc for sm_100a (cross-compiles without a GPU).

    python -m oxillama_b200.build [--verbose] [--force]
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
import warnings

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "_obj")
LIB = os.path.join(HERE, "libqk_cuda.so")
# Python extension over torch's C++ objects (csrc/qk_torch.cpp), for this Python and this torch alone; the package runs without it
EXT = os.path.join(HERE, "_qk_torch" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
SOURCES = ["qk_api.cu", "qk_simple.cu", "qk_gemv_mma.cu", "qk_gemv_imma.cu", "qk_dec_q80.cu", "qk_dec_q40.cu",
           "qk_dec_iq4xs.cu", "qk_dec_q6k.cu", "qk_dec_q5k.cu", "qk_dec_q3k.cu", "qk_dec_q2k.cu", "qk_noalloc.cu", "qk_gemm_tc.cu", "qk_tc_q4k.cu", "qk_tc_q4k_wide.cu", "qk_tc_q80.cu", "qk_tc_q40.cu", "qk_tc_q6k.cu", "qk_tc_q6k_wide.cu", "qk_tc_iq4xs.cu", "qk_moe.cu", "qk_moe_q4k.cu", "qk_moe_q80.cu", "qk_moe_q40.cu", "qk_moe_iq4xs.cu", "qk_moe_q6k.cu", "qk_gather.cu", "qk_gguf.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def _newer(src_list, target):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(s) > t for s in src_list)


def _ext_command(src):
    import torch
    base = os.path.dirname(torch.__file__)
    inc = [sysconfig.get_paths()["include"], os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
           os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")]
    lib = os.path.join(base, "lib")
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DQK_TORCH_VERSION="{torch.__version__}"',
            *(f"-I{i}" for i in inc), src, "-o", EXT,
            f"-L{lib}", f"-Wl,-rpath,{lib}", "-ltorch_python", "-ltorch_cpu", "-lc10_cuda", "-lc10"]


def _build_extension(force: bool = False) -> None:
    """Builds EXT where it is missing, older than its source or made by another command (another torch, another Python).
    Without torch, its headers, Python's or a C++ compiler there is none, and an old one is not left behind: calls then go
    through ctypes."""
    src, stamp = os.path.join(CSRC, "qk_torch.cpp"), os.path.join(OBJ, os.path.basename(EXT) + ".cmd")
    try:
        cmd = _ext_command(src)
        made_by = " ".join([sys.version, *cmd])
        if not force and not _newer([src], EXT) and os.path.exists(stamp) and open(stamp).read() == made_by:
            return
        subprocess.check_call(cmd)
        with open(stamp, "w") as f:
            f.write(made_by)
    except (ImportError, AttributeError, OSError, subprocess.CalledProcessError) as e:
        warnings.warn(f"the Python extension {os.path.basename(EXT)} was not built, device calls go through ctypes: {e!r}")
        if os.path.exists(EXT):
            os.remove(EXT)
    untagged = os.path.join(os.path.dirname(EXT), "_qk_torch.so")  # a name that any Python would import
    if untagged != EXT and os.path.exists(untagged):
        os.remove(untagged)


def build(verbose: bool = False, force: bool = False) -> str:
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    os.makedirs(OBJ, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(os.path.dirname(HERE), "include", "qk_cuda.h"))
    objs, jobs = [], []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _newer([s] + headers, o):
            cmd = [nvcc, *NVCC_FLAGS, "-c", s, "-o", o]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
                print(" ".join(cmd), flush=True)
            jobs.append(cmd)
    if jobs:  # the translation units are independent: compile them side by side
        from concurrent.futures import ThreadPoolExecutor
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 1)) as pool:
            list(pool.map(subprocess.check_call, jobs))
    if force or _newer(objs, LIB):
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.check_call(cmd)
    _build_extension(force)
    return LIB


if __name__ == "__main__":
    print(build(verbose="--verbose" in sys.argv, force="--force" in sys.argv))
