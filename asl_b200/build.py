"""Build recipe for libaslb.so (CUDA, sm_100a) in-tree.

Each .cu under csrc/ is compiled to an object in parallel, then linked into
asl_b200/libaslb.so. Objects are only rebuilt when a source or header is newer.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
OBJ = PKG / "_build"
LIB = PKG / "libaslb.so"

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-O3",
              "--expt-relaxed-constexpr", "-I", str(ROOT / "include"), "-I", str(CSRC)]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found")


def _sources() -> list[Path]:
    """The longest compilations first (two to four minutes each for D3Q27 and D3Q19)."""
    return sorted(CSRC.glob("*.cu"), key=lambda p: ("_q27_" not in p.name, "_q19_" not in p.name, p.name))


def _headers() -> list[Path]:
    return sorted(list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + list((ROOT / "include").glob("*.h")))


def _stale(target: Path, deps: list[Path]) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def _file_flags(src: Path) -> list[str]:
    """The collision writes every multiply-add itself (csrc/collide.cuh), so that all its kernels round alike; contraction
    would fuse some of its packed products into sums."""
    return ["--fmad=false"] if src.name.startswith(("step_", "batch_")) else []


def _compile(src: Path, extra: list[str], verbose: bool) -> Path:
    out = OBJ / (src.stem + ".o")
    if not _stale(out, [src] + _headers()):
        return out
    cmd = [nvcc(), *ARCH, *NVCC_FLAGS, *_file_flags(src), *extra, "-c", str(src), "-o", str(out)]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    return out


def build(verbose: bool = False, ptxas_info: bool = False) -> Path:
    """Compile every CUDA source for sm_100a and link libaslb.so. Returns its path."""
    OBJ.mkdir(exist_ok=True)
    extra = ["-Xptxas", "-v"] if ptxas_info else []
    srcs = _sources()
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(lambda s: _compile(s, extra, verbose), srcs))
    if _stale(LIB, objs):
        cmd = [nvcc(), *ARCH, "-shared", "-o", str(LIB), *map(str, objs), "-lcudart"]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.run(cmd, check=True)
    return LIB


if __name__ == "__main__":
    build(verbose=True, ptxas_info="--ptxas" in sys.argv)
