"""Build ``libaxtb_gpu.so`` in-tree for sm_100a (``python -m axtb_b200.build``)."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

HERE = Path(__file__).resolve().parent
SRC = HERE / "csrc" / "axtb_gpu.cu"
TRD = HERE / "csrc" / "trd.cu"  # the tridiagonal reduction's kernels: their own unit, compiled beside the engine
OUT = HERE / "libaxtb_gpu.so"
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
         "-shared"]


def nvcc() -> str:
    for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and Path(c).exists():
            return c
    raise RuntimeError("nvcc not found")


def sources():
    return [SRC, TRD] + sorted((HERE / "csrc").glob("*.cuh")) + [HERE / "csrc" / "trd_classes.h"] + [HERE / "csrc" / "params" / "gfn2_tables.h"] + \
        sorted((HERE.parent / "include").glob("*.h"))


def build(force: bool = False) -> Path:
    if not force and OUT.exists() and OUT.stat().st_mtime >= max(p.stat().st_mtime for p in sources()):
        return OUT
    tmp = OUT.with_suffix(".so.tmp")
    objs = [OUT.parent / (p.stem + ".o") for p in (SRC, TRD)]
    flags = [f for f in FLAGS if f != "-shared"]
    jobs = [subprocess.Popen([nvcc(), *flags, "-c", "-o", str(o), str(p)]) for p, o in zip((SRC, TRD), objs)]
    for job in jobs:
        job.wait()
    for job in jobs:
        if job.returncode:
            raise subprocess.CalledProcessError(job.returncode, job.args)
    subprocess.run([nvcc(), *FLAGS, "-o", str(tmp), *map(str, objs)], check=True)
    for o in objs:
        o.unlink()
    tmp.replace(OUT)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv))
