"""Build recipe for libmlstm_b200.so (plain nvcc, sm_100a only) and for _host.so, the native host side of the PyTorch
functions (plain g++ against the installed PyTorch); both in-tree next to this file.

    python -m mlstm_kernels_b200.build          # incremental
    python -m mlstm_kernels_b200.build --force  # rebuild everything

nvcc cross-compiles without a GPU.  Objects go to mlstm_kernels_b200/build/ (git-ignored).
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libmlstm_b200.so")
HOST = os.path.join(PKG, "_host.so")
SOURCES = ["api.cu", "gates.cu", "step.cu", "chunkwise_simt.cu", "chunkwise_sm100.cu", "chunkwise_bw_sm100.cu", "noalloc.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--use_fast_math=false", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found: the CUDA toolkit is required to build libmlstm_b200.so")
    return cand


def _deps_mtime() -> float:
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hdrs.append(os.path.join(os.path.dirname(PKG), "include", "mlstm_b200.h"))
    return max(os.path.getmtime(h) for h in hdrs)


def _host_command() -> list[str]:
    import torch
    from torch.utils import cpp_extension

    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [*cpp_extension.include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{p}" for p in inc),
            os.path.join(CSRC, "host.cpp"), "-o", HOST, f"-L{PKG}", "-l:libmlstm_b200.so", "-Wl,-rpath,$ORIGIN",
            f"-L{lib}", "-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"]


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    hdr_t = _deps_mtime()
    jobs = []
    objs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ, src.replace(".cu", ".o"))
        objs.append(o)
        if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hdr_t):
            flags = [f for f in NVCC_FLAGS if f != "--use_fast_math=false"]
            cmd = [nvcc, *flags, "-c", s, "-o", o]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    if jobs:
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 1)) as ex:
            for out in ex.map(run, jobs):
                if verbose and out:
                    print(out)
    if jobs or not os.path.exists(LIB):
        run([nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcuda"])
    host_src = os.path.join(CSRC, "host.cpp")
    if force or not os.path.exists(HOST) or os.path.getmtime(HOST) < max(os.path.getmtime(host_src), hdr_t):
        run(_host_command())
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
