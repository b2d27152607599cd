"""Build liblgs.so (the CUDA prover library) in-tree for sm_100a with nvcc.

Each translation unit under csrc/ is compiled to an object in csrc/_build/ (in parallel), then
linked into ligesis_b200/liblgs.so.  Rebuilds only what is older than its sources/headers.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = CSRC / "_build"
LIB = PKG / "liblgs.so"
INCLUDE = PKG.parent / "include"

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ARCH + [
    "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall",
    "--expt-relaxed-constexpr", "-Xcompiler", "-pthread", "-I", str(CSRC), "-I", str(INCLUDE),
]

# Host code whose time depends on where the linker puts it, which any edit elsewhere moves: the loops
# of the C entry points that reduce an input's words (12 % of lgs_subset_sum_hash on 128 x 4096, 1.15
# or 1.30 ms) and the verifier's functions (2^7 x 2^17: 7.8 or 8.1 ms; its loops are better left as
# they fall inside an aligned function).
FILE_FLAGS = {
    "capi.cu": ["-Xcompiler", "-falign-functions=64", "-Xcompiler", "-falign-loops=64"],
    "verify.cpp": ["-Xcompiler", "-falign-functions=64"],
}


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found: the prover library needs the CUDA toolkit to build")


def _sources() -> list[Path]:
    return sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cpp")])


def _headers() -> list[Path]:
    return sorted([*CSRC.glob("*.cuh"), *CSRC.glob("*.hpp"), *INCLUDE.glob("*.h")])


def _compile(nvcc: str, src: Path, obj: Path, extra: list[str]) -> None:
    flags = [*NVCC_FLAGS, *FILE_FLAGS.get(src.name, []), *extra]
    if src.suffix == ".cpp":
        flags += ["-x", "cu"]
    cmd = [nvcc, *flags, "-c", str(src), "-o", str(obj)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src.name}:\n{res.stdout}\n{res.stderr}")


def build(verbose: bool = False, force: bool = False, extra: list[str] | None = None) -> Path:
    nvcc = _nvcc()
    extra = list(extra or [])
    OBJ.mkdir(exist_ok=True)
    hdr_mtime = max((h.stat().st_mtime for h in _headers()), default=0.0)
    todo = []
    objs = []
    for src in _sources():
        obj = OBJ / (src.stem + ".o")
        objs.append(obj)
        if force or not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, hdr_mtime):
            todo.append((src, obj))
    with cf.ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        futs = [ex.submit(_compile, nvcc, s, o, extra) for s, o in todo]
        for f in futs:
            f.result()
    if todo or not LIB.exists() or LIB.stat().st_mtime < max(o.stat().st_mtime for o in objs):
        cmd = [nvcc, *ARCH, "-shared", "-Xcompiler", "-fPIC", "-o", str(LIB), *map(str, objs),
               "-lpthread"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    if verbose:
        print(f"built {LIB} ({len(todo)} objects recompiled)")
    return LIB


if __name__ == "__main__":
    build(verbose=True, force="--force" in sys.argv)
