"""Build libbmc_b200.so for sm_100a, in-tree (next to the Python package that loads it).

    python bmc-jax_b200/build.py [--force] [-v]

nvcc cross-compiles without a GPU. The translation units compile in parallel into _build/ (bmc_impl.cu once
per pool count) and are linked into one library, which is rebuilt when any source under csrc/ or the public
header is newer than it; only objects older than the sources they come from are recompiled.
"""
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
SRC = HERE / "csrc"
OBJ = HERE / "_build"
OUT = HERE / "bmc_b200" / "libbmc_b200.so"
HEADER = HERE.parent / "include" / "bmc_b200.h"
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
         "-Xcompiler", "-fPIC,-O2", "--expt-relaxed-constexpr"]
MAX_CEST = 5
ALONE = {"bmc_mlp.cu"}          # includes none of the other sources


def units():
    """(object name, source, extra flags) of every translation unit, the slowest first."""
    per_nc = [(f"bmc_impl_{n}.o", SRC / "bmc_impl.cu", [f"-DBMC_NC={n}"]) for n in range(MAX_CEST, -1, -1)]
    return per_nc + [(p.stem + ".o", p, []) for p in sorted(SRC.glob("*.cu")) if p.name != "bmc_impl.cu"]


def sources():
    return sorted(SRC.glob("*.cu")) + sorted(SRC.glob("*.cuh")) + sorted(SRC.glob("*.h")) + [HEADER]


def stale() -> bool:
    return not OUT.exists() or any(p.stat().st_mtime > OUT.stat().st_mtime for p in sources())


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not stale():
        return OUT
    OBJ.mkdir(exist_ok=True)
    shared = [p for p in sources() if p.suffix != ".cu"]

    def compile_one(unit):
        name, src, extra = unit
        obj = OBJ / name
        deps = [src, HEADER] if src.name in ALONE else [src, *shared]
        if not force and obj.exists() and all(p.stat().st_mtime <= obj.stat().st_mtime for p in deps):
            return obj
        cmd = [NVCC, *FLAGS, *extra, *(["-Xptxas", "-v"] if verbose else []), "-c", "-o", str(obj), str(src)]
        print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.stdout:
            print(r.stdout, flush=True)
        if r.returncode:
            obj.unlink(missing_ok=True)
            raise subprocess.CalledProcessError(r.returncode, cmd)
        return obj

    with ThreadPoolExecutor(os.cpu_count() or 1) as pool:
        objs = list(pool.map(compile_one, units()))
    tmp = OUT.with_suffix(".so.tmp")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", str(tmp), *map(str, objs)],
                   check=True)
    os.replace(tmp, OUT)
    return OUT


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print("built", OUT)
