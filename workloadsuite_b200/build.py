"""Build the sm_100a shared library ``lib/libssd_b200.so`` in-tree with nvcc, and, where PyTorch is installed,
``lib/ssd_b200_torch.so``, the short way from PyTorch tensors to it, with the host compiler.

    python -m workloadsuite_b200.build [--force] [--verbose]
    python workloadsuite_b200/build.py [--force] [--verbose]      (the library alone needs no PyTorch)

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
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
LIB_DIR = PKG / "lib"
LIB = LIB_DIR / "libssd_b200.so"
TORCH_LIB = LIB_DIR / "ssd_b200_torch.so"
STAMP = LIB_DIR / "libssd_b200.stamp"
TORCH_STAMP = LIB_DIR / "ssd_b200_torch.stamp"
BINDING = CSRC / "torch_binding.cpp"
HEADER = ROOT / "include" / "ssd_b200.h"

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


def _hash(files, *extra: str) -> str:
    h = hashlib.sha256()
    for f in sorted(files):
        h.update(f.name.encode())
        h.update(f.read_bytes())
    for e in extra:
        h.update(e.encode())
    return h.hexdigest()


def _fingerprint() -> str:
    """What the library was built from."""
    return _hash([f for f in CSRC.glob("*") if f != BINDING] + [HEADER], " ".join(NVCC_FLAGS))


def _torch():
    """PyTorch, or None where it is not installed."""
    try:
        import torch
    except ImportError:
        return None
    return torch


def _torch_flags(torch):
    return ["-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]


def _torch_fingerprint(torch) -> str:
    """What the binding was built from and against: it holds inline code of one PyTorch's C++ headers and one Python's."""
    return _hash([BINDING, HEADER], " ".join(_torch_flags(torch)), torch.__version__, str(sysconfig.get_config_var("EXT_SUFFIX")))


def source_fingerprint() -> str:
    """Hash of the sources of the dominant kernel (the two-head tensor-core kernel and the headers it includes) and of
    the compiler flags: what an ncu summary of that kernel must have been captured from to describe the kernel that
    runs now."""
    h = hashlib.sha256()
    for name in ("ssd_tc2.cu", "tile_walk.cuh", "tc_common.cuh", "tc_ptx.cuh", "ssd_common.cuh"):
        h.update(name.encode())
        h.update((CSRC / name).read_bytes())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def _stamped(lib: Path, stamp: Path, fingerprint: str) -> bool:
    return lib.exists() and stamp.exists() and stamp.read_text().strip() == fingerprint


def is_current() -> bool:
    torch = _torch()
    return _stamped(LIB, STAMP, _fingerprint()) and (
        torch is None or _stamped(TORCH_LIB, TORCH_STAMP, _torch_fingerprint(torch)))


def _start_torch_binding(torch):
    """Compiles ``csrc/torch_binding.cpp`` (a CPython module on PyTorch's C++ API) in the background."""
    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    cmd = [os.environ.get("CXX") or shutil.which("g++") or "c++", *_torch_flags(torch),
           "-I", str(HEADER.parent), "-I", str(root / "include"), "-I", str(root / "include/torch/csrc/api/include"),
           "-I", str(cuda / "include"), "-I", sysconfig.get_paths()["include"], str(BINDING), "-o", str(TORCH_LIB),
           "-L", str(root / "lib"), f"-Wl,-rpath,{root / 'lib'}", "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _finish(jobs, verbose: bool) -> bool:
    """Waits for compilations [(source, process)]; True if all went well."""
    good = True
    for src, pr in jobs:
        out, _ = pr.communicate()
        if pr.returncode != 0:
            good = False
            sys.stderr.write(f"--- compilation failed: {src.name}\n{out}\n")
        elif verbose or out.strip():
            sys.stderr.write(f"--- {src.name}\n{out}\n")
    return good


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every ``csrc/*.cu`` for sm_100a and link ``libssd_b200.so``; then the binding, where there is a PyTorch to
    bind to.  A binding that does not compile is an error, but leaves the library complete."""
    LIB_DIR.mkdir(exist_ok=True)
    torch = _torch()
    binding = None
    if torch is not None and (force or not _stamped(TORCH_LIB, TORCH_STAMP, _torch_fingerprint(torch))):
        TORCH_STAMP.unlink(missing_ok=True)
        binding = _start_torch_binding(torch)
    if force or not _stamped(LIB, STAMP, _fingerprint()):
        nvcc = _nvcc()
        objs = []
        jobs = []
        for src in sources():
            obj = LIB_DIR / (src.stem + ".o")
            cmd = [nvcc, *NVCC_FLAGS, "-I", str(HEADER.parent), "-I", str(CSRC), "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
            jobs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
            objs.append(obj)
        if not _finish(jobs, verbose):
            if binding is not None:
                binding.communicate()
            raise RuntimeError("compilation failed")
        link = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a",
                "-lcudart_static", "-lcuda", "-Xcompiler", "-fPIC"]
        subprocess.run(link, check=True)
        STAMP.write_text(_fingerprint())
    if binding is not None:
        if not _finish([(BINDING, binding)], verbose):
            raise RuntimeError("compilation of the PyTorch binding failed (the library itself is built)")
        TORCH_STAMP.write_text(_torch_fingerprint(torch))
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
