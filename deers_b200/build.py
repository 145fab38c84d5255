"""Builds ``libdeers_b200.so`` in-tree with nvcc for sm_100a.

These are the same commands a ``build.rs`` on the deers side would run.  Usage: ``python -m deers_b200.build [--force] [--verbose]``.
"""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIB_DIR, "libdeers_b200.so")
HOST_SRC = os.path.join(CSRC, "host_ext.cpp")
HOST_EXT = os.path.join(LIB_DIR, "_deers_host.so")      # native host layer of the Python mirror (ops.py)
SOURCES = ["ctx.cu", "attn_f32.cu", "attn_f32_few32.cu", "attn_f32_few64.cu", "attn_f32_few96.cu", "attn_f32_few128.cu", "umma_selftest.cu", "attn_fwd_f16_sm100.cu", "attn_bwd_f16_sm100.cu",
           "rope_pack.cu", "optim.cu", "rmsnorm.cu", "attn_decode.cu", "gemm_f16_sm100.cu", "gemm_f16x3_sm100.cu", "gemm_f32.cu",
           "gemm_f32_loose.cu", "gemm_f32_tc.cu", "gemm_f32_tc_loose.cu", "gpt_ops.cu", "gpt_model.cu", "comm.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC,-fvisibility=hidden", "--use_fast_math=false"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIB_DIR, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(HERE, "..", "include", "deers_b200.h"))
    objs = []
    procs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(LIB_DIR, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + headers):
            cmd = [_nvcc()] + [f for f in NVCC_FLAGS if not f.startswith("--use_fast_math")] + \
                  (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, pr in procs:
        out, _ = pr.communicate()
        if pr.returncode != 0 or verbose:
            sys.stderr.write(f"--- {src}\n{out}\n")
        failed |= pr.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    if force or procs or _stale(LIB, objs):
        cmd = [_nvcc(), "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a",
                                                       "-Xcompiler", "-fPIC", "-cudart", "static"]
        subprocess.run(cmd, check=True)
    return LIB


def build_host(force: bool = False, verbose: bool = False) -> str:
    """The CPython extension ops.py calls: host code only, linked against the library above and torch."""
    header = os.path.join(HERE, "..", "include", "deers_b200.h")
    if not force and not _stale(HOST_EXT, [HOST_SRC, header]):
        return HOST_EXT
    import sysconfig

    import torch
    t = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    cmd = ["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f"-I{t}/include",
           f"-I{t}/include/torch/csrc/api/include", f"-I{cuda}/include", f"-I{sysconfig.get_paths()['include']}", HOST_SRC,
           "-o", HOST_EXT, f"-L{LIB_DIR}", "-ldeers_b200", f"-L{t}/lib", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
           "-ltorch", "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    out = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if out.returncode != 0 or verbose:
        sys.stderr.write(f"--- host_ext.cpp\n{out.stdout}\n")
    if out.returncode != 0:
        raise RuntimeError("g++ failed")
    return HOST_EXT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
    print(build_host(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
