"""Build liblesgpu.so (sm_100a) in-tree with nvcc.

Each translation unit compiles in its own nvcc process; the objects are
linked into ``new_repo_b200/liblesgpu.so`` next to this file.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
BUILD = HERE.parent / "_build"
LIB = HERE / "liblesgpu.so"
SOURCES = ["spectral_inst.cu", "spectral_xfwd.cu", "spectral_xinv.cu", "spectral_xinv_f64.cu", "spectral_ypass.cu", "spectral_ypass_f64.cu", "solver.cu", "capi.cu", "mlp.cu", "noalloc.cu"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
# The device code is linked as it is: a process's first state loads the images of
# four or five source files, each 11 ms to unpack where it is compressed and 1-4 ms
# where it is not (first FP64 / mixed state of a process 43 / 58 ms and 23 / 30 ms;
# the library grows from 37 to 81 MB).
FLAGS = ["--compress-mode=none", "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-fno-strict-aliasing",
         "--expt-relaxed-constexpr", "-I", str(HERE.parent / "include")]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found")


def _stale(obj: Path, src: Path) -> bool:
    if not obj.exists():
        return True
    deps = [src, Path(__file__)] + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.hpp")) + ([src.with_name(src.name.replace("_f64", ""))] if "_f64" in src.name else []) + [HERE.parent / "include" / "lesgpu.h"]
    t = obj.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps if d.exists())


def build(verbose: bool = False, ptxas_info: bool = False) -> Path:
    BUILD.mkdir(exist_ok=True)
    srcs = [CSRC / s for s in SOURCES if (CSRC / s).exists()]
    objs = [BUILD / (s.stem + ".o") for s in srcs]
    cc = nvcc()

    def compile_one(pair):
        src, obj = pair
        if not _stale(obj, src) and not ptxas_info:
            return ""
        cmd = [cc, *ARCH, *FLAGS, "-c", str(src), "-o", str(obj)]
        if ptxas_info:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stderr}")
        return r.stderr

    with ThreadPoolExecutor(max_workers=len(srcs)) as ex:
        logs = list(ex.map(compile_one, zip(srcs, objs)))
    if verbose:
        for l in logs:
            if l:
                print(l)
    if not LIB.exists() or any(o.stat().st_mtime > LIB.stat().st_mtime for o in objs):
        # link to a temporary name and rename: a process loading the library
        # meanwhile sees the old file or the new one, never a partial one
        tmp = LIB.with_name(LIB.name + ".tmp")
        cmd = [cc, *ARCH, "-shared", "-o", str(tmp), *map(str, objs), "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stderr}")
        os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(verbose=True, ptxas_info="-v" in sys.argv))
