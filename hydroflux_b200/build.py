"""Build the sm_100a shared library hydroflux_b200/libhydroflux_gpu.so.

nvcc cross-compiles without a GPU. Floating-point flags keep the kernels'
rounding identical to the reference's Rust f64 code: no FMA contraction,
IEEE-rounded division and square root.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
ROOT = os.path.dirname(HERE)
INCLUDE = os.path.join(ROOT, "include")
OUT = os.path.join(HERE, "libhydroflux_gpu.so")

SOURCES = ["hf_kernels.cu", "hf_tiles.cu", "hf_dual.cu", "hf_api.cu", "hf_noalloc.cu", "hf_batch.cu",
           "hf_serve.cu", "hf_adjoint.cu", "hf_calib.cu", "hf_io.cu"]
# hf_tiles.cu is compiled once more for each other tile geometry (the default
# macros give 32 x 8 tiles by 256 threads; see hf_internal.h).
GEOMETRIES = [("hf_tiles.cu", "hf_tiles_%s.o" % name,
               ["-DHF_GEOM=" + name, "-DHF_GEOM_INDEX=%d" % index, "-DHF_TILE_Y=%d" % rows,
                "-DHF_THREADS=%d" % threads, "-DHF_MIN_BLOCKS=%d" % blocks])
              for name, index, rows, threads, blocks in (
                  ("g32", 1, 32, 1024, 1), ("g8w", 2, 8, 768, 1), ("g8m", 3, 8, 384, 2),
                  ("g4", 4, 4, 512, 1))]
GEOMETRIES.append(("hf_dual.cu", "hf_dual_g8d.o",
                   ["-DHF_GEOM=g8d", "-DHF_GEOM_INDEX=5", "-DHF_TILE_Y=8", "-DHF_THREADS=512",
                    "-DHF_MIN_BLOCKS=1"]))
GENCODE = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ["-O3", "-std=c++17", "-lineinfo", "--fmad=false", "-prec-div=true",
              "-prec-sqrt=true", "-Xcompiler", "-fPIC", "-Xcompiler", "-O2",
              "--expt-relaxed-constexpr"]


def nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _deps():
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    files.append(os.path.join(INCLUDE, "hydroflux_gpu.h"))
    files.append(os.path.abspath(__file__))
    return files


def needs_build() -> bool:
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    return any(os.path.getmtime(f) > t for f in _deps())


def build(force: bool = False, verbose: bool = False) -> str:
    if not (force or needs_build()):
        return OUT
    objdir = os.path.join(HERE, "_build")
    os.makedirs(objdir, exist_ok=True)
    units = [(src, src.replace(".cu", ".o"), []) for src in SOURCES] + GEOMETRIES
    objs, procs = [], []
    for src, name, defs in units:  # the translation units compile in parallel
        obj = os.path.join(objdir, name)
        cmd = [nvcc(), *GENCODE, *NVCC_FLAGS, *defs, "-I", INCLUDE, "-c",
               os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((cmd, subprocess.Popen(cmd)))
        objs.append(obj)
    failed = [cmd for cmd, p in procs if p.wait() != 0]
    if failed:
        raise subprocess.CalledProcessError(1, failed[0])
    tmp = OUT + ".tmp"
    subprocess.run([nvcc(), *GENCODE, "-shared", "-cudart", "static", "-o", tmp, *objs, "-lz"],
                   check=True)
    os.replace(tmp, OUT)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
