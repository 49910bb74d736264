"""Builds ``libgturbo_gb.so`` in-tree with nvcc for sm_103a.

Translation units are compiled in parallel into ``gturbo3d_gb300/_build/`` and
linked into ``gturbo3d_gb300/libgturbo_gb.so`` (both git-ignored).  A unit is
recompiled when its source or any header in ``csrc/`` or ``include/`` is newer
than its object file.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
BUILD = PKG / "_build"
LIB = PKG / "libgturbo_gb.so"

ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
NVCC_FLAGS = ["-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
              "-Xptxas", "-v"] + ARCH
HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-fno-fast-math", "-ffp-contract=off"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found: the CUDA toolkit is required to build gturbo3d_gb300")


def _newest_header() -> float:
    hs = list(CSRC.glob("*.h")) + list(CSRC.glob("*.cuh")) + list((ROOT / "include").glob("*.h"))
    return max((h.stat().st_mtime for h in hs), default=0.0)


def _compile(src: Path, nvcc: str, hdr_time: float, verbose: bool) -> tuple[Path, str]:
    obj, log = BUILD / (src.name + ".o"), BUILD / (src.name + ".log")
    if obj.exists() and log.exists() and obj.stat().st_mtime >= max(src.stat().st_mtime, hdr_time):
        return obj, ""
    if src.suffix == ".cu":
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
    else:
        # host-only C++: plain IEEE arithmetic (no contraction) so the set-up
        # tables and forcing draws match the CPU restatement bit for bit
        cmd = [nvcc, "-ccbin", "g++", "-x", "c++", "-Xcompiler", ",".join(HOST_FLAGS), "-c", str(src),
               "-o", str(obj)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"compile failed: {' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
    log.write_text(r.stdout + r.stderr)   # registers and spills of every kernel, for the resource tests
    return obj, (r.stdout + r.stderr) if verbose else ""


def build(verbose: bool = False) -> Path:
    nvcc = _nvcc()
    BUILD.mkdir(exist_ok=True)
    srcs = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cpp"))
    hdr = _newest_header()
    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        results = list(ex.map(lambda s: _compile(s, nvcc, hdr, verbose), srcs))
    objs = [o for o, _ in results]
    if verbose:
        for _, log in results:
            if log:
                print(log)
    newest = max(o.stat().st_mtime for o in objs)
    if not LIB.exists() or LIB.stat().st_mtime < newest:
        tmp = LIB.with_suffix(".so.tmp")
        cmd = [nvcc, "-shared", *ARCH, "-o", str(tmp), *map(str, objs)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed: {' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
        os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv))
