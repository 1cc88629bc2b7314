"""Builds libjvpfa.so in-tree with nvcc for sm_100a.

Usage: ``python -m jvp_flash_attention_b200.build [--force] [--verbose]``.
Each ``csrc/*.cu`` is compiled to an object file under ``csrc/_obj`` (in parallel) and the
objects are linked into ``jvp_flash_attention_b200/libjvpfa.so``.  A translation unit is rebuilt
only when it or a header is newer than its object.  ``csrc/native.cpp``, the host side of a call
(``_native.so``, a Python extension module linked against torch and libjvpfa.so), is built with g++, again also when
the command or the version of torch is another one than it was built with.
"""
from __future__ import annotations

import argparse
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
OBJ = CSRC / "_obj"
LIB = PKG_DIR / "libjvpfa.so"
NATIVE = PKG_DIR / "_native.so"
NATIVE_STAMP = OBJ / "native.stamp"  # what the present _native.so was built with
INCLUDE = PKG_DIR.parent / "include"

NVCC_FLAGS = [
    "-std=c++17",
    "-O3",
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-Xcompiler",
    "-fPIC",
    "--expt-relaxed-constexpr",
    "-I",
    str(INCLUDE),
    *os.environ.get("JVPFA_EXTRA_NVCC_FLAGS", "").split(),
]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"
    return cand if Path(cand).exists() else "nvcc"


def _newest_header() -> float:
    hs = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + list(INCLUDE.glob("*.h"))
    return max(h.stat().st_mtime for h in hs)


def _native_cmd() -> list[str]:
    import torch
    from torch.utils import cpp_extension

    torch_lib = Path(torch.__file__).parent / "lib"
    return [
        os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-DTORCH_EXTENSION_NAME=_native",
        "-I", str(INCLUDE), "-I", str(CSRC / "compat"), "-I", sysconfig.get_paths()["include"],
        *(f"-isystem{p}" for p in cpp_extension.include_paths("cuda")),
        str(CSRC / "native.cpp"), "-o", str(NATIVE),
        f"-L{torch_lib}", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10",
        f"-L{PKG_DIR}", "-l:libjvpfa.so", "-Wl,-rpath,$ORIGIN",
    ]


def _native_with() -> str:
    import torch

    return "\n".join([f"torch {torch.__version__}", f"python {sys.version}", *_native_cmd()])


def _native_stale() -> bool:
    sources = [CSRC / "native.cpp", INCLUDE / "jvpfa.h", *(CSRC / "compat").rglob("*.hpp")]
    if not NATIVE.exists() or NATIVE.stat().st_mtime < max(f.stat().st_mtime for f in sources):
        return True
    return not NATIVE_STAMP.exists() or NATIVE_STAMP.read_text() != _native_with()


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every CUDA source for sm_100a and link the shared library; returns its path."""
    OBJ.mkdir(exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    hdr_time = _newest_header()
    jobs = []
    for src in sources:
        obj = OBJ / (src.stem + ".o")
        stale = force or not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, hdr_time)
        if stale:
            cmd = [_nvcc(), *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    if jobs:
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as ex:
            for cmd, r in ex.map(run, jobs):
                if verbose or r.returncode != 0:
                    sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
                if r.returncode != 0:
                    raise RuntimeError(f"nvcc failed for {cmd[-3]}")
    objs = [str(OBJ / (s.stem + ".o")) for s in sources]
    if jobs or not LIB.exists():
        cmd = [_nvcc(), "-shared", "-o", str(LIB), *objs, "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    if force or _native_stale():
        r = subprocess.run(_native_cmd(), capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("g++ failed for native.cpp")
        NATIVE_STAMP.write_text(_native_with())
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
