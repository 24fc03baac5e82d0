"""Compile the CUDA sources into the in-tree C-ABI shared library (sm_100a only), and the small C++ module through
which eager PyTorch calls reach it."""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PACKAGE_DIR = Path(__file__).resolve().parent
CSRC_DIR = PACKAGE_DIR / "csrc"
LIB_DIR = PACKAGE_DIR / "_lib"
LIB_PATH = LIB_DIR / "libternel_b200.so"

# Host functions begin on a cache line, so that their speed does not follow what else is in the library: the worker that packs blocks
# lost 12% (5120x5120 codes on eight cores 925 -> 1036 us) when it came to begin 48 bytes into one, and has it back.
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-falign-functions=64", "-shared",
]


BINDING_SOURCE = CSRC_DIR / "torch_binding.cpp"
BINDING_PATH = LIB_DIR / "_ternel_torch.so"

CHECKED_LIB_PATH = LIB_DIR / "libternel_b200_checked.so"
# The checked build: every global store tests its index first and records a violation instead of writing
# (the record is one device array shared by all source files, hence relocatable device code).
CHECKED_FLAGS = ["-DTQ1_BOUNDS_CHECK", "-rdc=true"]


def sources() -> list[Path]:
    return sorted(CSRC_DIR.glob("*.cu"))


def _nvcc() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(found).exists():
        raise RuntimeError("nvcc not found; the library can only be built with the CUDA toolkit")
    return found


def is_stale(target: Path = LIB_PATH) -> bool:
    if not target.exists():
        return True
    built = target.stat().st_mtime
    deps = sources() + list(CSRC_DIR.glob("*.cuh")) + [PACKAGE_DIR.parent / "include" / "ternel_b200.h", Path(__file__)]
    return any(p.stat().st_mtime > built for p in deps)


def build_checked(force: bool = False) -> Path:
    """Build ``_lib/libternel_b200_checked.so``, the bounds-checking variant used by tests/test_gpu_bounds.py."""
    return build(force=force, target=CHECKED_LIB_PATH, extra=CHECKED_FLAGS)


def build(force: bool = False, verbose: bool = False, target: Path = LIB_PATH, extra: "list[str] | None" = None) -> Path:
    """Build ``_lib/libternel_b200.so`` (or ``target``) when missing or older than a source file."""
    if not force and not is_stale(target):
        return target
    LIB_DIR.mkdir(exist_ok=True)
    tmp = LIB_DIR / f".{target.stem}.{os.getpid()}.so"
    cmd = [_nvcc(), *NVCC_FLAGS, *(extra or []), *( ["-Xptxas", "-v"] if verbose else [] ),
           "-o", str(tmp), *map(str, sources())]
    done = subprocess.run(cmd, capture_output=True, text=True)
    if done.returncode != 0:
        tmp.unlink(missing_ok=True)
        raise RuntimeError(f"nvcc failed:\n{done.stdout}\n{done.stderr}")
    if verbose:
        print(done.stderr)
    os.replace(tmp, target)
    return target


def binding_target() -> str:
    """What the eager call path has to be built for: its C++ side follows one PyTorch and one Python."""
    import torch

    return f"torch {torch.__version__}, {sys.implementation.cache_tag}"


def binding_built_for() -> "str | None":
    """What the module in ``_lib`` was built for, None where there is none (or none that says so)."""
    stamp = BINDING_PATH.with_suffix(".target")
    return stamp.read_text() if BINDING_PATH.exists() and stamp.exists() else None


def binding_is_stale() -> bool:
    header = PACKAGE_DIR.parent / "include" / "ternel_b200.h"
    return binding_built_for() != binding_target() or any(
        p.stat().st_mtime > BINDING_PATH.stat().st_mtime for p in (BINDING_SOURCE, header))


def build_binding(force: bool = False) -> Path:
    """Build ``_lib/_ternel_torch.so``, the eager call path, against the installed PyTorch (host code only)."""
    if not force and not binding_is_stale():
        return BINDING_PATH
    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    LIB_DIR.mkdir(exist_ok=True)
    tmp = LIB_DIR / f".{BINDING_PATH.stem}.{os.getpid()}.so"
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           "-isystem", str(root / "include"), "-isystem", str(root / "include/torch/csrc/api/include"),
           "-isystem", str(cuda / "include"), "-isystem", sysconfig.get_paths()["include"],
           str(BINDING_SOURCE), "-o", str(tmp), f"-L{root / 'lib'}", "-ltorch_python", "-ltorch", "-ltorch_cpu",
           "-ltorch_cuda", "-lc10", "-lc10_cuda", f"-L{cuda / 'lib64'}", "-lcudart", f"-Wl,-rpath,{root / 'lib'}"]
    done = subprocess.run(cmd, capture_output=True, text=True)
    if done.returncode != 0:
        tmp.unlink(missing_ok=True)
        raise RuntimeError(f"g++ failed:\n{done.stdout}\n{done.stderr}")
    os.replace(tmp, BINDING_PATH)
    BINDING_PATH.with_suffix(".target").write_text(binding_target())
    return BINDING_PATH


if __name__ == "__main__":
    print(build(force=True, verbose=True))
    print(build_binding(force=True))
