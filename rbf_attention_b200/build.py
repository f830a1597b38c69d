"""Builds librbf_b200.so in-tree with nvcc for sm_100a (no torch headers, no libcuda link dependency) and _host.so, the
CPython extension on top of it that ops.py calls (torch headers).

Usage: ``python -m rbf_attention_b200.build [--force] [--verbose]``.
"""

from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "librbf_b200.so")
HOST = os.path.join(HERE, "_host.so")
HOST_SOURCE = os.path.join(CSRC, "host.cpp")
HOST_STAMP = os.path.join(HERE, "_host.stamp")      # the torch and interpreter that _host.so was built for
C_HEADER = os.path.join(os.path.dirname(HERE), "include", "rbf_b200.h")
SOURCES = ["capi.cu", "rbf_prep.cu", "rbf_fwd.cu", "rbf_fwd_tf32.cu", "rbf_bwd.cu", "rbf_bwd_fused.cu",
           "rbf_bwd_fused128.cu", "ce_loss.cu", "layer_norm.cu", "col_sums.cu", "gelu.cu", "narrow.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cand = os.path.join(cuda_home, "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _headers() -> list[str]:
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))] + [C_HEADER]


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _host_command() -> list[str]:
    """g++ on host.cpp against the installed torch, linked to the library beside it."""
    import torch

    root = os.path.dirname(torch.__file__)
    includes = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"), sysconfig.get_paths()["include"]]
    # the compiler that nvcc takes for host code: one with a C++ runtime of its own does not mix with torch's libraries
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            f'-DRBF_TORCH_VERSION="{torch.__version__}"', *(f"-I{i}" for i in includes), HOST_SOURCE,
            "-o", HOST, f"-L{os.path.join(root, 'lib')}", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lc10",
            "-lc10_cuda", f"-L{HERE}", "-l:librbf_b200.so", "-Wl,-rpath,$ORIGIN"]


def _host_target() -> str:
    """torch's C++ interface belongs to one version of it: another torch (or interpreter) wants another extension."""
    import torch

    return f"torch {torch.__version__}, {sys.implementation.cache_tag}\n"


def _host_stale() -> bool:
    if _stale(HOST, [HOST_SOURCE, C_HEADER]) or not os.path.exists(HOST_STAMP):
        return True
    with open(HOST_STAMP) as f:
        return f.read() != _host_target()


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles every translation unit to an object, links the shared library and builds the extension. Returns the
    library's path."""
    headers = _headers()
    objs = []
    jobs = []
    for src in SOURCES:
        obj = os.path.join(CSRC, src.replace(".cu", ".o"))
        objs.append(obj)
        if force or _stale(obj, [os.path.join(CSRC, src), *headers]):
            cmd = [_nvcc(), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"build failed: {' '.join(cmd)}")

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as pool:
        list(pool.map(run, jobs))
    if jobs or force or _stale(LIB, objs):
        run([_nvcc(), "-shared", "-o", LIB, *objs, "-lcudart"])
    if force or _host_stale():
        run(_host_command())
        with open(HOST_STAMP, "w") as f:
            f.write(_host_target())
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
