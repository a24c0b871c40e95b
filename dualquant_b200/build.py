"""Builds libdualquant_b200.so (sm_100a only, nvcc) and the torch binding _torch_host.so (g++), in-tree.

Usage: python -m dualquant_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_DIR = os.path.join(PKG_DIR, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libdualquant_b200.so")
HOST_SOURCE = "torch_host.cpp"
HOST_PATH = os.path.join(LIB_DIR, "_torch_host.so")

SOURCES = [
    "dq_runtime.cu",
    "weights_int4.cu",
    "bcd.cu",
    "act_quant_int4.cu",
    "act_quant_had_bf16.cu",
    "act_quant_had_f32.cu",
    "quant_fp4.cu",
    "gemm_w4a4_int4.cu",
    "gemm_w4a4_int4_tm.cu",
    "gemv_w4a4_int4.cu",
    "gemv_w4a4_int4_fused.cu",
    "gemm_fp4.cu",
    "linear_w4a4.cu",
    "mma_peak.cu",
    "gemm_a16w4.cu",
    "decoder_ops.cu",
    "gemm_w4a4_int4_f8.cu",
    "gemm_w4a4_int4_f8_out0.cu",
    "gemm_w4a4_int4_f8_out1.cu",
    "gemm_w4a4_int4_f8_out2.cu",
    "gemm_w4a4_int4_f8_out3.cu",
    "gemm_w4a4_int4_f8_out5.cu",
    "gemm_fp4_persist.cu",
    "exchange.cu",
]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--fmad=true",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _newest_source_mtime() -> float:
    newest = 0.0
    for root in (CSRC, os.path.join(PKG_DIR, "..", "include")):
        for name in os.listdir(root):
            newest = max(newest, os.path.getmtime(os.path.join(root, name)))
    return newest


def needs_build() -> bool:
    newest = _newest_source_mtime()
    return any(not os.path.exists(p) or os.path.getmtime(p) < newest for p in (LIB_PATH, HOST_PATH))


def _host_command() -> list:
    """The binding against this interpreter's torch; its symbols come from the torch that is already loaded
    when the module is imported."""
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths, library_paths

    cuda = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")
    dirs = [*include_paths(), sysconfig.get_paths()["include"], cuda]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *(f"-isystem{d}" for d in dirs), os.path.join(CSRC, HOST_SOURCE), "-o", HOST_PATH,
            *(f"-L{d}" for d in library_paths()), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
            "-ltorch_python", "-ldl"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ into one shared library, and the torch binding next to it; returns the
    library's path."""
    if not force and not needs_build():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(LIB_DIR, src.replace(".cu", ".o"))
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), flush=True)
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    procs.append((HOST_SOURCE, subprocess.Popen(_host_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                                                text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- {src}\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("the compiler failed; see output above")
    link = [_nvcc(), "-shared", "-o", LIB_PATH, *objs, "-gencode", "arch=compute_100a,code=sm_100a",
            "-Xcompiler", "-fPIC"]
    subprocess.run(link, check=True)
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
