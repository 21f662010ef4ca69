"""In-tree build of the CUDA library: nvcc -> pypto_b200/libpypto_b200.so (sm_100a only), and of the native host path of
the operators in front of it: g++ -> pypto_b200/_native.so (a CPython module over torch's C++ headers).

The shared object links the CUDA runtime statically and resolves the one driver symbol it needs
(cuTensorMapEncodeTiled) at run time, so it loads on a machine without a GPU driver.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libpypto_b200.so"
SOURCES = ["capi.cu", "li_score.cu", "topk_select.cu", "sfa_decode.cu", "sfa_pair.cu", "sfa_slice.cu", "prolog.cu", "prolog_gemm.cu",
           "prolog_sgemm.cu", "prolog_wide.cu"]
HEADERS = [CSRC / "common.cuh", CSRC / "sfa_common.cuh", PKG.parent / "include" / "pypto_b200.h"]


NATIVE = PKG / "_native.so"
NATIVE_SOURCE = CSRC / "native.cpp"


def nvcc_path() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found (set $NVCC)")


def needs_build() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    deps = [CSRC / s for s in SOURCES] + HEADERS
    return any(d.stat().st_mtime > t for d in deps)


def build_native(force: bool = False) -> Path:
    """The module links the CUDA library next to it and torch's own libraries (loaded by `import torch` before it)."""
    deps = (NATIVE_SOURCE, LIB, PKG.parent / "include" / "pypto_b200.h")
    if not force and NATIVE.exists() and all(d.stat().st_mtime <= NATIVE.stat().st_mtime for d in deps):
        return NATIVE
    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(nvcc_path()).resolve().parent.parent
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-isystem", str(root / "include"),
           "-isystem", str(root / "include" / "torch" / "csrc" / "api" / "include"), "-isystem", str(cuda / "include"),
           "-isystem", sysconfig.get_paths()["include"], str(NATIVE_SOURCE), "-o", str(NATIVE), str(LIB),
           "-Wl,-rpath,$ORIGIN", "-L", str(root / "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    subprocess.run(cmd, check=True)
    return NATIVE


def build(force: bool = False, verbose: bool = False) -> Path:
    _build_library(force, verbose)
    build_native(force)
    return LIB


def _build_library(force: bool, verbose: bool) -> Path:
    if not force and not needs_build():
        return LIB
    objs = []
    bdir = PKG / "build"
    bdir.mkdir(exist_ok=True)
    common = [nvcc_path(), "-std=c++17", "-O3", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a",
              "-Xcompiler", "-fPIC", "-Xptxas", "-v" if verbose else "-warn-spills"]
    procs = []
    for s in SOURCES:
        obj = bdir / (Path(s).stem + ".o")
        objs.append(str(obj))
        procs.append((s, subprocess.Popen(common + ["-c", str(CSRC / s), "-o", str(obj)], stdout=subprocess.PIPE,
                                          stderr=subprocess.STDOUT, text=True)))
    failed = False
    for s, pr in procs:
        out, _ = pr.communicate()
        if pr.returncode != 0 or verbose:
            sys.stderr.write(f"--- {s}\n{out}\n")
        failed |= pr.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    link = [nvcc_path(), "-shared", "-Xlinker", "-soname=libpypto_b200.so", "-cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(LIB)] + objs + ["-ldl"]
    subprocess.run(link, check=True)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
