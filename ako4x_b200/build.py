"""Builds ``lib/libako4x_b200.so`` from ``csrc/*.cu`` with nvcc for sm_100a, and the Python binding
module ``lib/_native*.so`` from ``csrc/bindings.cpp`` with the host compiler against PyTorch's headers.

Run as ``python -m ako4x_b200.build`` (add ``--force`` to rebuild everything, ``-v`` for the
ptxas resource report). The library is built in-tree; nothing is installed.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIBDIR = PKG / "lib"
OBJDIR = PKG / "lib" / "obj"
LIB = LIBDIR / "libako4x_b200.so"
INCLUDE = PKG.parent / "include"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-I", str(INCLUDE),
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put /usr/local/cuda/bin on PATH")


def _headers_mtime() -> float:
    hs = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + list(INCLUDE.glob("*.h"))
    return max((h.stat().st_mtime for h in hs), default=0.0)


def build(force: bool = False, verbose: bool = False) -> Path:
    nvcc = _nvcc()
    OBJDIR.mkdir(parents=True, exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    if not sources:
        raise RuntimeError(f"no .cu sources under {CSRC}")
    hdr_m = _headers_mtime()
    jobs = []
    for src in sources:
        obj = OBJDIR / (src.stem + ".o")
        if force or not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, hdr_m):
            cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append((src, cmd))

    def run(job):
        src, cmd = job
        p = subprocess.run(cmd, capture_output=True, text=True)
        return src, p.returncode, p.stdout + p.stderr

    failed = []
    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for src, rc, out in ex.map(run, jobs):
            if verbose or rc != 0:
                sys.stderr.write(f"--- {src.name}\n{out}\n")
            if rc != 0:
                failed.append(src.name)
    if failed:
        raise RuntimeError(f"nvcc failed for: {', '.join(failed)}")
    objs = [str(OBJDIR / (s.stem + ".o")) for s in sources]
    if jobs or not LIB.exists():
        cmd = [nvcc, "-shared", "-o", str(LIB), *objs]
        p = subprocess.run(cmd, capture_output=True, text=True)
        if p.returncode != 0:
            raise RuntimeError("link failed:\n" + p.stdout + p.stderr)
    build_native(force)
    return LIB


def build_native(force: bool = False) -> Path:
    """The binding module; rebuilt when its source, the C-ABI header or PyTorch itself is newer."""
    import torch
    from ._cabi import NATIVE_PATH as out
    src = CSRC / "bindings.cpp"
    troot = Path(torch.__file__).resolve().parent
    newest = max(p.stat().st_mtime for p in (src, INCLUDE / "ako4x_b200.h", troot / "version.py"))
    if not force and out.exists() and out.stat().st_mtime >= newest:
        return out
    cuda = Path(_nvcc()).resolve().parents[1]
    tlib = troot / "lib"
    cmd = [os.environ.get("CXX") or "g++", "-std=c++17", "-O2", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", str(INCLUDE), "-I", sysconfig.get_paths()["include"], "-I", str(troot / "include"),
           "-I", str(troot / "include" / "torch" / "csrc" / "api" / "include"), "-I", str(cuda / "include"),
           str(src), "-o", str(out), "-L", str(LIBDIR), "-lako4x_b200", "-Wl,-rpath,$ORIGIN",
           "-L", str(tlib), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"]
    p = subprocess.run(cmd, capture_output=True, text=True)
    if p.returncode != 0:
        raise RuntimeError("building the binding module failed:\n" + p.stdout + p.stderr)
    return out


if __name__ == "__main__":
    lib = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(lib)
