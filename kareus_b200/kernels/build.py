"""Ahead-of-time build of ``libkareus_b200.so`` with nvcc for sm_100a.

All kernels are compiled in-tree (no runtime JIT: the reference compiles its collective kernels to
PTX at run time, ``3rdparty/mscclpp/python/mscclpp/utils.py:85-127``).  The library exposes a
plain C ABI, so it has no dependency on PyTorch headers and builds in seconds without a GPU.
``_fastcall.so`` (``csrc/torch/fastcall.cpp``) is the extension module between PyTorch tensors and that ABI
for the calls whose host time counts.  It needs g++ and the headers of Python and PyTorch (15 s more); the library works
without it, with more host time a call, so where it cannot be built that is a warning.

    python -m kareus_b200.kernels.build          # build if sources are newer than the library
    python -m kareus_b200.kernels.build --force
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
import warnings
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path
from typing import List

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
OBJ = HERE / "build"
LIB = HERE / "libkareus_b200.so"
FASTCALL_SRC = CSRC / "torch" / "fastcall.cpp"
FASTCALL_DEPS = (FASTCALL_SRC, CSRC / "native_calls.h")
FASTCALL = HERE / "_fastcall.so"

ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ["-O3", "-std=c++17", "-lineinfo", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC"
              ]


def nvcc() -> str:
    for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and Path(c).exists():
            return c
    raise RuntimeError("nvcc not found; set NVCC or install the CUDA toolkit")


def sources() -> List[Path]:
    return sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cpp")))


def _digest() -> str:
    h = hashlib.sha256()
    for p in sorted(CSRC.iterdir()):
        if p.suffix in (".cu", ".cuh", ".h", ".cpp"):
            h.update(p.name.encode())
            h.update(p.read_bytes())
    h.update(" ".join(ARCH_FLAGS + NVCC_FLAGS).encode())
    return h.hexdigest()


def is_current() -> bool:
    stamp = OBJ / "digest"
    return LIB.exists() and stamp.exists() and stamp.read_text() == _digest()


def _fastcall_digest() -> str:
    import torch
    h = hashlib.sha256(b"".join(p.read_bytes() for p in FASTCALL_DEPS))
    h.update(f"{torch.__version__} {sysconfig.get_config_var('SOABI')}".encode())
    return h.hexdigest()


def build_fastcall(force: bool = False) -> Path:
    """The extension module; needs the library to link against."""
    stamp = OBJ / "fastcall.digest"
    digest = _fastcall_digest()
    if not force and FASTCALL.exists() and stamp.exists() and stamp.read_text() == digest:
        return FASTCALL
    import torch
    root = Path(torch.__file__).resolve().parent
    cuda_inc = Path(nvcc()).resolve().parent.parent / "include"
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wno-attributes",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DKB_TORCH_VERSION="{torch.__version__}"',
           "-I", str(root / "include"), "-I", str(root / "include/torch/csrc/api/include"),
           "-I", sysconfig.get_paths()["include"], "-I", str(cuda_inc), str(FASTCALL_SRC), "-o", str(FASTCALL),
           "-L", str(root / "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda",
           "-L", str(HERE), "-l:" + LIB.name, "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {FASTCALL_SRC.name}:\n{r.stdout}\n{r.stderr}")
    stamp.write_text(digest)
    return FASTCALL


def _build_fastcall_or_warn(force: bool = False) -> None:
    try:
        build_fastcall(force)
    except (ImportError, OSError, RuntimeError) as e:
        FASTCALL.unlink(missing_ok=True)          # one of other sources or another PyTorch is worse than none
        warnings.warn(f"{FASTCALL.name} was not built, calls take more host time: {e}", RuntimeWarning, stacklevel=3)


def _compile(src: Path, verbose: bool) -> Path:
    obj = OBJ / (src.stem + ".o")
    cmd = [nvcc(), *ARCH_FLAGS, *NVCC_FLAGS, "-I", str(CSRC), "-c", str(src), "-o", str(obj)]
    if src.suffix == ".cpp":
        cmd.insert(1, "-x")
        cmd.insert(2, "cu")
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
    if verbose:
        sys.stderr.write(r.stderr)
    return obj


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and is_current():
        _build_fastcall_or_warn()
        return LIB
    OBJ.mkdir(exist_ok=True)
    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 2)) as ex:
        objs = list(ex.map(lambda s: _compile(s, verbose), sources()))
    cmd = [nvcc(), *ARCH_FLAGS, "-shared", "-o", str(LIB), *map(str, objs), "-cudart", "shared"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    (OBJ / "digest").write_text(_digest())
    _build_fastcall_or_warn(force)
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
