"""Build liblemoq_b200.so (the C-ABI library) in-tree with nvcc for sm_100a, and the Python binding of its short operators.

    python leanmoe-quant_b200/csrc/build.py [--verbose]

The library has no dependency on torch or Python: it links against the CUDA runtime
only.  ``lemoq/_bind.so`` (bind.cpp, g++) links against the library, torch and Python.  Objects are rebuilt when a source or header is newer than the object.
"""

from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))
SOURCES = ["cabi.cu", "gemv_w8.cu", "stream_gemv.cu", "moe_grouped.cu", "attn_decode.cu", "small_ops.cu", "step.cu", "step_tile.cu", "batched_w8.cu", "ep_exchange.cu",
           "w8_gemm.cu", "w8_pair.cu", "attn_i8.cu", "prompt.cu", "prompt_ops.cu", "prompt_attn.cu"]
HEADERS = ["common.cuh", "gemv_common.cuh", "stream.cuh", "stream_gemv.cuh", "step_kernel.h", "step_route.h", "kernels.h", "tc.cuh", "w8_tile.cuh", "prompt.h", os.path.join(ROOT, "include", "lemoq_b200.h")]
LIB = os.path.join(HERE, "liblemoq_b200.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
] + os.environ.get("LEMOQ_NVCC_EXTRA", "").split()


def _newer(src: str, dst: str) -> bool:
    return not os.path.exists(dst) or os.path.getmtime(src) > os.path.getmtime(dst)


BIND_SOURCE, BIND = os.path.join(HERE, "bind.cpp"), os.path.join(os.path.dirname(HERE), "lemoq", "_bind.so")


def build_bind(verbose: bool = False) -> str:
    """The binding for the running interpreter and its torch; it finds the library next to it (rpath)."""
    import sysconfig

    import torch

    if not any(_newer(src, BIND) for src in (BIND_SOURCE, HEADERS[-1], __file__)):
        return BIND
    root = os.path.dirname(torch.__file__)
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
               os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI), *("-isystem" + d for d in include), BIND_SOURCE, "-o", BIND, LIB,
           "-Wl,-rpath,$ORIGIN/../csrc", "-L" + os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError("g++ failed for %s" % BIND_SOURCE)
    return BIND


def build(verbose: bool = False) -> str:
    deps = [h if os.path.isabs(h) else os.path.join(HERE, h) for h in HEADERS]
    objs, jobs = [], []
    for s in SOURCES:
        src = os.path.join(HERE, s)
        obj = os.path.join(HERE, s.replace(".cu", ".o"))
        objs.append(obj)
        if _newer(src, obj) or any(_newer(d, obj) for d in deps) or _newer(__file__, obj):
            cmd = [NVCC, *FLAGS, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with ThreadPoolExecutor(max_workers=max(1, min(len(jobs), os.cpu_count() or 1))) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError("nvcc failed for %s" % cmd[-3])
    if jobs or not os.path.exists(LIB):
        cmd = [NVCC, "-shared", "-o", LIB, *objs, "-cudart", "static", "-Xlinker", "-soname=liblemoq_b200.so"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    build_bind(verbose)
    return LIB


if __name__ == "__main__":
    print(build(verbose="--verbose" in sys.argv))
