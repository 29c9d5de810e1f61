"""Builds the sm_100a shared library ``hfem_b200/libhfem_b200.so`` in-tree."""
from __future__ import annotations

import os
import subprocess
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libhfem_b200.so")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
              "-Xcompiler", "-fPIC", "-diag-suppress", "177"]
# element shapes (nd, npv, npf, ngv, ngf) of launch.cuh's HFEM_SHAPES, one translation unit each
SHAPES = [(2, 3, 2, 3, 2), (2, 6, 3, 6, 3), (2, 10, 4, 12, 4), (2, 15, 5, 16, 5), (3, 4, 3, 4, 3), (3, 10, 6, 14, 6),
          (3, 20, 10, 24, 12)]


def _stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(SRC, f) for f in os.listdir(SRC) if f.endswith((".cu", ".cuh", ".h"))]
    deps.append(os.path.join(HERE, "..", "include", "hfem_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return LIB
    nvcc = os.environ.get("NVCC", "nvcc")
    flags = [*NVCC_FLAGS, *(["-Xptxas=-v"] if verbose else [])]
    with tempfile.TemporaryDirectory() as tmp:
        jobs = [(os.path.join(SRC, "hfem_capi.cu"), [], os.path.join(tmp, "capi.o"))]
        jobs += [(os.path.join(SRC, "shape.cu"), [f"-DHFEM_{k}={v}" for k, v in zip(("ND", "NPV", "NPF", "NGV", "NGF"), s)], os.path.join(tmp, f"shape{i}.o"))
                 for i, s in enumerate(SHAPES)]
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 1)) as ex:
            # list(): a failed compile raises here
            list(ex.map(lambda j: subprocess.run([nvcc, *flags, *j[1], "-c", "-o", j[2], j[0]], check=True), jobs))
        subprocess.run([nvcc, *NVCC_FLAGS, "-shared", "-o", LIB + ".tmp", *[j[2] for j in jobs]], check=True)
    os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    print(build(force=True, verbose=True))
