"""Build ``libnanoquant_b200.so`` in-tree with nvcc for sm_100a.

This replaces the reference's ``compile_kernel.sh`` / ``setup.py`` (a torch
CUDAExtension built for the local GPU): the library here has a plain C ABI, no
torch or Python headers, and is cross-compiled for sm_100a whether or not a GPU
is present.  ``_nq_torch.so`` beside it is the host path between PyTorch and that ABI
(``csrc/nq_torch.cpp``, plain C++ against the installed torch).  Usage: ``python -m nanoquant_b200.build [--force] [--verbose]``.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libnanoquant_b200.so")
EXT_PATH = os.path.join(PKG_DIR, "_nq_torch.so")
EXT_SOURCE = "nq_torch.cpp"
INCLUDE = os.path.join(os.path.dirname(PKG_DIR), "include")

SOURCES = ["nq_core.cu", "nq_pack.cu", "nq_gemv.cu", "nq_gemm.cu", "nq_wgemm.cu", "nq_pgemm.cu", "nq_batch.cu", "nq_comm.cu", "nq_dense.cu", "nq_probe.cu"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--expt-relaxed-constexpr", "--extended-lambda",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: set NVCC or put the CUDA toolkit on PATH")


def _stale() -> bool:
    if not os.path.exists(LIB_PATH) or not os.path.exists(EXT_PATH):
        return True
    t = min(os.path.getmtime(LIB_PATH), os.path.getmtime(EXT_PATH))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(INCLUDE, "nanoquant_b200.h"),
                                                                  os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def _ext_compile(obj: str) -> list:
    import sysconfig
    import torch
    from torch.utils import cpp_extension
    inc = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], INCLUDE,
                                           os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    return ["g++", "-std=c++17", "-O2", "-fPIC", "-fvisibility=hidden", "-Wall", "-Wno-sign-compare",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *[a for d in inc for a in ("-isystem", d)], "-c", os.path.join(CSRC, EXT_SOURCE), "-o", obj]


def _ext_link(obj: str) -> list:
    import torch
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    return ["g++", "-shared", "-o", EXT_PATH, obj, "-L", PKG_DIR, "-l:libnanoquant_b200.so", "-L", lib, "-ltorch_python",
            "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10_cuda", "-lc10", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every ``csrc/*.cu`` into one shared library and the torch host path into another; returns the
    library's path."""
    if not force and not _stale():
        return LIB_PATH
    nvcc = _nvcc()
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(CSRC, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), flush=True)
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    ext_obj = os.path.join(CSRC, EXT_SOURCE.replace(".cpp", ".o"))
    procs.append((EXT_SOURCE, subprocess.Popen(_ext_compile(ext_obj), stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                                               text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if out.strip() and (verbose or p.returncode != 0):
            print(out, flush=True)
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed, see output above")
    link = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-lcudart"]
    subprocess.run(link, check=True)
    subprocess.run(_ext_link(ext_obj), check=True)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
