"""Builds the native code in-tree (sm_100a only):

    python -m dlblas_b200.build [--force] [--verbose]

    dlblas_b200/_dlblas_b200.so   the CUDA library: a C ABI (include/dlblas_b200.h) that links against neither torch nor
                                  Python (nvcc)
    dlblas_b200/_host.so          the host side of the operators, a CPython extension on torch's C++ API that calls that
                                  C ABI (g++)

No JIT at import time.
"""
import argparse
import os
import subprocess
import sys

from ._C import HOST_PATH, host_is_current, host_tag

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OUT = os.path.join(PKG, "_dlblas_b200.so")
SOURCES = ["abi.cu", "sort.cu", "quant.cu", "route.cu", "p2p.cu", "gemm_fp8.cu", "gemm_bf16.cu"]
HEADERS = ["common.cuh", "sort.cuh", "tile_width.h", "umma.cuh", os.path.join("..", "..", "include", "dlblas_b200.h")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
]


HOST_SOURCE = "host.cpp"


def _host_command(obj_source, out):
    import sysconfig

    import torch
    root = os.path.dirname(os.path.abspath(torch.__file__))
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    lib = os.path.join(root, "lib")
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    return (["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-Wall", "-Wextra",
             f"-D_GLIBCXX_USE_CXX11_ABI={abi}", f'-DDLB_HOST_TAG="{host_tag()}"'] +
            [f for d in inc for f in ("-isystem", d)] + [obj_source, "-o", out, "-L" + lib, "-Wl,-rpath," + lib,
             "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"])


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    objdir = os.path.join(PKG, "build")
    os.makedirs(objdir, exist_ok=True)
    hdrs = [os.path.normpath(os.path.join(CSRC, h)) for h in HEADERS]
    objs, procs = [], []
    host = os.path.join(CSRC, HOST_SOURCE)
    # torch's C++ interface is not stable: another torch, another build
    if force or _stale(HOST_PATH, [host, hdrs[-1]]) or not host_is_current(HOST_PATH):
        procs.append((HOST_SOURCE, subprocess.Popen(_host_command(host, HOST_PATH), stdout=subprocess.PIPE,
                                                    stderr=subprocess.STDOUT, text=True)))
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(objdir, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + hdrs):
            cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if out.strip():                # errors and warnings; the registers of every kernel with `verbose`
            sys.stderr.write(f"--- {src} ---\n{out}\n")
        failed = failed or p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed while building the dlblas_b200 extension")
    if force or procs or _stale(OUT, objs):
        cmd = [_nvcc(), "-shared", "-o", OUT] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stdout)
    return OUT


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
