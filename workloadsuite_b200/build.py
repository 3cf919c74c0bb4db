"""Build the sm_100a shared library ``lib/libssd_b200.so`` in-tree with nvcc, and ``lib/ssd_b200_torch.so``, the
short way from PyTorch tensors to it, with the host compiler.

    python -m workloadsuite_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU.  The library is a plain C-ABI ``.so``
(``include/ssd_b200.h``); it does not link against PyTorch, the small binding module does.
"""
from __future__ import annotations

import argparse
import hashlib
import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
LIB_DIR = PKG / "lib"
LIB = LIB_DIR / "libssd_b200.so"
TORCH_LIB = LIB_DIR / "ssd_b200_torch.so"
STAMP = LIB_DIR / "libssd_b200.stamp"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; set NVCC or add the CUDA toolkit to PATH")


def sources():
    return sorted(CSRC.glob("*.cu"))


def _fingerprint() -> str:
    h = hashlib.sha256()
    for f in sorted(list(CSRC.glob("*")) + [ROOT / "include" / "ssd_b200.h"]):
        h.update(f.name.encode())
        h.update(f.read_bytes())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def source_fingerprint() -> str:
    """Hash of the sources of the dominant kernel (the two-head tensor-core kernel and the headers it includes) and of
    the compiler flags: what an ncu summary of that kernel must have been captured from to describe the kernel that
    runs now."""
    h = hashlib.sha256()
    for name in ("ssd_tc2.cu", "tc_common.cuh", "tc_ptx.cuh", "ssd_common.cuh"):
        h.update(name.encode())
        h.update((CSRC / name).read_bytes())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def is_current() -> bool:
    return LIB.exists() and TORCH_LIB.exists() and STAMP.exists() and STAMP.read_text().strip() == _fingerprint()


def _start_torch_binding():
    """Compiles ``csrc/torch_binding.cpp`` (a CPython module on PyTorch's C++ API) in the background."""
    import sysconfig

    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    cmd = [os.environ.get("CXX") or shutil.which("g++") or "c++", "-O2", "-std=c++17", "-shared", "-fPIC",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", str(ROOT / "include"), "-I", str(root / "include"), "-I", str(root / "include/torch/csrc/api/include"),
           "-I", str(cuda / "include"), "-I", sysconfig.get_paths()["include"],
           str(CSRC / "torch_binding.cpp"), "-o", str(TORCH_LIB),
           "-L", str(root / "lib"), f"-Wl,-rpath,{root / 'lib'}", "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every ``csrc/*.cu`` for sm_100a and link ``libssd_b200.so``."""
    if not force and is_current():
        return LIB
    LIB_DIR.mkdir(exist_ok=True)
    nvcc = _nvcc()
    objs = []
    procs = []
    for src in sources():
        obj = LIB_DIR / (src.stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-I", str(ROOT / "include"), "-I", str(CSRC), "-c", str(src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    failed = False
    procs.append((CSRC / "torch_binding.cpp", _start_torch_binding()))
    for src, pr in procs:
        out, _ = pr.communicate()
        if pr.returncode != 0:
            failed = True
            sys.stderr.write(f"--- compilation failed: {src.name}\n{out}\n")
        elif verbose or out.strip():
            sys.stderr.write(f"--- {src.name}\n{out}\n")
    if failed:
        raise RuntimeError("compilation failed")
    link = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a",
            "-lcudart_static", "-lcuda", "-Xcompiler", "-fPIC"]
    subprocess.run(link, check=True)
    STAMP.write_text(_fingerprint())
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
