"""Build recipe of the in-tree shared library ``libcudafoam.so`` (sm_100a).

Cross-compiles without a GPU: ``python -m metal4foam_b200.build``.
"""
from __future__ import annotations

import os
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libcudafoam.so")
SOURCES = ["cf_context.cu", "cf_solve.cu", "cf_batched.cu", "cf_adjoint.cu", "cf_static.cu",
           "cf_multi.cu", "cf_tune.cu",
           "cf_persist.cu", "cf_cluster.cu", "cf_amg.cu", "cf_many.cu", "cf_check.cu",
           "cf_coupled.cu", "cf_partition.cu", "cf_resident.cu", "cf_clupcg.cu",
           "cf_clubicg.cu", "cf_resbicg.cu"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def sources():
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def _stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = sources() + [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(ROOT, "include", "cudafoam.h"))
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu of csrc/ into libcudafoam.so for sm_100a."""
    if not force and not _stale():
        return LIB
    flags = ["-O3", "-std=c++17", *ARCH, "-lineinfo", "-Xcompiler", "-fPIC",
             "-I", os.path.join(ROOT, "include"), "-I", CSRC]
    if verbose:
        flags.insert(0, "-Xptxas=-v")

    def run(cmd):
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
            raise RuntimeError("nvcc failed building libcudafoam.so")
        if verbose:
            sys.stderr.write(res.stderr)

    # one compiler per file at a time on every core, then the link
    with tempfile.TemporaryDirectory() as tmp:
        objs = [os.path.join(tmp, os.path.basename(s) + ".o") for s in sources()]
        with ThreadPoolExecutor(max(1, min(16, os.cpu_count() or 1))) as pool:
            list(pool.map(run, [[NVCC, *flags, "-c", "-o", o, s]
                                for o, s in zip(objs, sources())]))
        run([NVCC, *ARCH, "-Xcompiler", "-fPIC", "-shared", "-o", LIB + ".tmp", *objs])
    os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
