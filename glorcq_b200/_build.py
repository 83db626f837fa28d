"""In-tree build of libglorcq_b200.so with nvcc for sm_100a (cross-compiles without a GPU) and of the host path's
native module (csrc/native.cpp, against torch's headers) with the host compiler."""

from __future__ import annotations

import os
import subprocess
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libglorcq_b200.so")
NATIVE = os.path.join(HERE, "_native.so")
SOURCES = ["api.cu", "moe.cu", "attn.cu", "lm_head.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-shared", "-Xcompiler", "-fPIC", "--use_fast_math=false"]


def _stale(target, deps) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(d) > os.path.getmtime(target) for d in deps)


def _run(cmd) -> str:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(cmd[0] + " failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    return res.stderr


def _build_lib(verbose):
    srcs = [os.path.join(CSRC, s) for s in SOURCES]
    flags = [f for f in NVCC_FLAGS if not f.startswith("--use_fast_math")]
    out = _run([os.environ.get("NVCC", "nvcc")] + flags + ["--threads", "0"] + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB] + srcs)
    if verbose:
        print(out)


def _build_native():
    import torch
    from torch.utils.cpp_extension import CUDA_HOME, include_paths
    inc = include_paths() + [sysconfig.get_paths()["include"], os.path.join(CUDA_HOME or "/usr/local/cuda", "include")]
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    _run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + [f"-isystem{d}" for d in inc] +
         ["-o", NATIVE, os.path.join(CSRC, "native.cpp"), f"-L{libs}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
          "-ltorch_python"])


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile csrc/*.cu into glorcq_b200/libglorcq_b200.so and csrc/native.cpp into glorcq_b200/_native.so; returns the
    library path."""
    header = os.path.join(HERE, "..", "include", "glorcq_b200.h")
    cuda = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))] + [header]
    jobs = []
    if force or _stale(LIB, cuda):
        jobs.append(lambda: _build_lib(verbose))
    if force or _stale(NATIVE, [os.path.join(CSRC, "native.cpp"), header]):
        jobs.append(_build_native)
    with ThreadPoolExecutor(2) as pool:
        for f in [pool.submit(j) for j in jobs]:
            f.result()
    return LIB


if __name__ == "__main__":
    import sys
    print(build(force=True, verbose="-v" in sys.argv))
