"""Builds ``libcompactattn_b200.so`` in-tree with nvcc for sm_100a.

The library is plain CUDA C++ behind a C ABI (``include/compactattn_b200.h``); it links only the
static CUDA runtime, so it loads on a machine without a GPU driver (symbols can be inspected
there) and runs on a B200.

Usage: ``python -m compactattention_b200.build [--force] [--verbose]``

Development builds (cycle accounting, timing experiments) go to a separate file and never replace
the product library: ``python -m compactattention_b200.build --define CA_ATTN_PROFILE=1 --output
compactattention_b200/libcompactattn_b200_profile.so``.
"""
from __future__ import annotations

import argparse
import hashlib
import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_PATH = PKG_DIR / "libcompactattn_b200.so"
STAMP_PATH = PKG_DIR / "libcompactattn_b200.so.stamp"
CALLS_SOURCE = PKG_DIR / "binding" / "calls.cpp"
CALLS_PATH = PKG_DIR / "_calls.so"
CALLS_STAMP_PATH = PKG_DIR / "_calls.so.stamp"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-cudart", "static",
    "-shared",
]


HEADER = PKG_DIR.parent / "include" / "compactattn_b200.h"


def header_define() -> str:
    """The header's hash, compiled into the library and into the native wrappers: both hold its struct layouts, and
    ``ops._native()`` lets them work together only where the hashes are the same."""
    return "CA_HEADER_HASH=" + hashlib.sha256(HEADER.read_bytes()).hexdigest()[:16]


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _fingerprint() -> str:
    h = hashlib.sha256()
    files = sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + [HEADER])
    for f in files:
        h.update(f.name.encode())
        h.update(f.read_bytes())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; cannot build libcompactattn_b200.so")
    return nvcc


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every ``csrc/*.cu`` into one shared library, and the native wrappers that go with it; skip what is up to date."""
    path = _build_library(force, verbose)
    build_calls(force)
    return path


def _build_library(force: bool, verbose: bool) -> Path:
    fp = _fingerprint()
    if not force and LIB_PATH.exists() and STAMP_PATH.exists() and STAMP_PATH.read_text().strip() == fp:
        return LIB_PATH
    cmd = [find_nvcc(), *NVCC_FLAGS, f"-D{header_define()}"]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", str(LIB_PATH), *[str(s) for s in sources()]]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or proc.returncode != 0:
        sys.stderr.write(proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError(f"nvcc failed with exit code {proc.returncode}")
    STAMP_PATH.write_text(fp + "\n")
    return LIB_PATH


def build_calls(force: bool = False) -> Path:
    """Compile the native form of the tensor-level wrappers (``binding/calls.cpp``) for this Python and torch."""
    import sysconfig

    import torch

    h = hashlib.sha256()
    for f in (CALLS_SOURCE, HEADER):
        h.update(f.read_bytes())
    h.update(f"{torch.__version__} {sys.version}".encode())
    fp = h.hexdigest()
    if not force and CALLS_PATH.exists() and CALLS_STAMP_PATH.exists() and CALLS_STAMP_PATH.read_text().strip() == fp:
        return CALLS_PATH
    root = Path(torch.__file__).resolve().parent
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D{header_define()}",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f"-I{root / 'include'}",
           f"-I{root / 'include' / 'torch' / 'csrc' / 'api' / 'include'}", f"-I{sysconfig.get_paths()['include']}",
           "-o", str(CALLS_PATH), str(CALLS_SOURCE), f"-L{root / 'lib'}", "-ltorch_python", "-ltorch_cpu", "-lc10"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        sys.stderr.write(proc.stdout + proc.stderr)
        raise RuntimeError(f"g++ failed with exit code {proc.returncode}")
    CALLS_STAMP_PATH.write_text(fp + "\n")
    return CALLS_PATH


def build_variant(defines: list[str], output: Path, verbose: bool = False) -> Path:
    """Compile the same sources with extra ``-D`` macros into ``output`` (a development build)."""
    output = Path(output).resolve()
    if output == LIB_PATH:
        raise ValueError("a development build must not overwrite the product library")
    cmd = [find_nvcc(), *NVCC_FLAGS, f"-D{header_define()}", *[f"-D{d}" for d in defines]]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", str(output), *[str(s) for s in sources()]]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or proc.returncode != 0:
        sys.stderr.write(proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError(f"nvcc failed with exit code {proc.returncode}")
    return output


def main() -> None:
    ap = argparse.ArgumentParser(description=__doc__)
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    ap.add_argument("--define", action="append", default=[], help="extra macro NAME=VALUE (development build; needs --output)")
    ap.add_argument("--output", default=None, help="where a development build is written")
    args = ap.parse_args()
    if args.define or args.output:
        if not (args.define and args.output):
            ap.error("--define and --output go together")
        print(build_variant(args.define, Path(args.output), verbose=args.verbose))
    else:
        print(build(force=args.force, verbose=args.verbose))
        print(CALLS_PATH)


if __name__ == "__main__":
    main()
