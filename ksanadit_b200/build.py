"""Builds the CUDA kernels and their C ABI into ``ksanadit_b200/lib/libksana_b200.so`` (sm_100a only), and the C++ side of the
single calls (``host_call.cpp``, a CPython extension against torch's headers) into ``ksanadit_b200/lib/ksana_b200_host.<torch>.so``.
The latter is an accelerator: where it cannot be built, that is said and the library is built all the same.

Usage: ``python -m ksanadit_b200.build [--force]``.  nvcc cross-compiles without a GPU present.
"""

from __future__ import annotations

import concurrent.futures
import os
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIBDIR = os.path.join(PKG, "lib")
LIB = os.path.join(LIBDIR, "libksana_b200.so")
SOURCES = ["capi.cu", "rowwise_quant.cu", "fp8_gemm.cu", "fp8_gemm_split.cu", "sage_prepass.cu", "sage_attn.cu", "sage_attn_dual.cu", "elementwise.cu", "fused.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--use_fast_math=false",
]


def _nvcc():
    return os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc")


def _deps():
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hdrs.append(os.path.join(os.path.dirname(PKG), "include", "ksana_b200.h"))
    return hdrs


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def _host_command(src, target):
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) or "/usr/local/cuda"
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
               os.path.join(cuda, "include")]
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *("-I" + d for d in include), src, "-o", target, "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]


def build_host(force: bool = False, verbose: bool = False) -> bool:
    """Builds the extension for the torch that is installed.  False, and why on stderr, where that cannot be done."""
    src = os.path.join(CSRC, "host_call.cpp")
    try:
        from .native import host_path
        target = host_path()
        if not (force or _stale(target, [src] + _deps())):
            return True
        part = f"{target[:-3]}.{os.getpid()}.so"
        cmd = _host_command(src, part)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode == 0:
            os.replace(part, target)
            return True
        why = "compiler failed"
    except (ImportError, OSError) as e:
        why = str(e)
    sys.stderr.write(f"the C++ side of the single calls was not built ({why}): they go through Python\n")
    return False


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIBDIR, exist_ok=True)
    srcs = [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    flags = [f for f in NVCC_FLAGS if not f.startswith("--use_fast_math")]
    objs, jobs = [], []
    for s in srcs:
        src = os.path.join(CSRC, s)
        obj = os.path.join(LIBDIR, s.replace(".cu", ".o"))
        objs.append(obj)
        if force or _stale(obj, [src] + _deps()):
            cmd = [_nvcc()] + flags + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with concurrent.futures.ThreadPoolExecutor(max_workers=max(1, min(8, len(jobs) + 1))) as ex:
        host = ex.submit(build_host, force, verbose)
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError("compiler failed: " + " ".join(cmd))
    if jobs or force or _stale(LIB, objs):
        cmd = [_nvcc(), "-shared", "-o", LIB] + objs + ["-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    host.result()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
