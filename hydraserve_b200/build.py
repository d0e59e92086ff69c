"""Builds the native parts in-tree: ``python -m hydraserve_b200.build``.

``hydraserve_b200/lib/libhs_sampler.so``, the C-ABI CUDA library, is what
``hydraserve_b200._lib`` loads (nvcc cross-compiles for sm_100a without a GPU);
``hydraserve_b200/_host.<interpreter>.so`` is the Python extension with the host side of a step
(plain C++; Python 3.10 or newer, x86-64 or aarch64).
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
SOURCES = [PKG / "csrc" / "hs_api.cu"]
HEADERS = sorted((PKG / "csrc").glob("*.cuh")) + sorted((PKG / "csrc").glob("*.h")) + [ROOT / "include" / "hs_sampler.h"]
OUTPUT = PKG / "lib" / "libhs_sampler.so"
HOST_SOURCES = [PKG / "csrc" / "hs_host.cpp"]
HOST_HEADERS = [ROOT / "include" / "hs_sampler.h"]
# (named for the interpreter: another one builds its own)
HOST_OUTPUT = PKG / f"_host{sysconfig.get_config_var('EXT_SUFFIX')}"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared",
]
CXX_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    return "nvcc"


def _stale(output: Path, inputs) -> bool:
    if not output.exists():
        return True
    built = output.stat().st_mtime
    return any(p.stat().st_mtime > built for p in inputs)


def needs_build() -> bool:
    return _stale(OUTPUT, SOURCES + HEADERS)


def _run(cmd, output: Path, verbose: bool) -> None:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or proc.returncode != 0:
        sys.stderr.write(proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed building {output}")


def build_host(force: bool = False, verbose: bool = False) -> Path:
    if force or _stale(HOST_OUTPUT, HOST_SOURCES + HOST_HEADERS):
        # (written next to its place and moved there, so that a process importing it meanwhile
        # sees the old file or the new one)
        fresh = HOST_OUTPUT.with_suffix(f".so.{os.getpid()}")
        _run([os.environ.get("CXX", "g++"), *CXX_FLAGS, "-I", sysconfig.get_paths()["include"],
              "-o", str(fresh), *map(str, HOST_SOURCES)], HOST_OUTPUT, verbose)
        os.replace(fresh, HOST_OUTPUT)
    return HOST_OUTPUT


def build(force: bool = False, verbose: bool = False) -> Path:
    build_host(force, verbose)
    if not force and not needs_build():
        return OUTPUT
    OUTPUT.parent.mkdir(parents=True, exist_ok=True)
    cmd = [_nvcc(), *NVCC_FLAGS]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    _run([*cmd, "-o", str(OUTPUT), *map(str, SOURCES)], OUTPUT, verbose)
    return OUTPUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
