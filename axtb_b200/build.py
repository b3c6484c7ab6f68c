"""Build ``libaxtb_gpu.so`` in-tree for sm_100a (``python -m axtb_b200.build``)."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import tempfile
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
    # objects and library in a folder of this call's own: several processes may build at once, each its own
    # whole library, the last of which stays
    with tempfile.TemporaryDirectory(prefix=".build", dir=OUT.parent) as work:
        objs = [Path(work) / (p.stem + ".o") for p in (SRC, TRD)]
        flags = [f for f in FLAGS if f != "-shared"]
        jobs = [subprocess.Popen([nvcc(), *flags, "-c", "-o", str(o), str(p)]) for p, o in zip((SRC, TRD), objs)]
        for job in jobs:
            job.wait()
        for job in jobs:
            if job.returncode:
                raise subprocess.CalledProcessError(job.returncode, job.args)
        tmp = Path(work) / OUT.name
        subprocess.run([nvcc(), *FLAGS, "-o", str(tmp), *map(str, objs)], check=True)
        tmp.replace(OUT)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv))
