"""Out of memory while a mesh is split over the SMs, on any of the host
threads, is an error that the caller handles, never the end of the process."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.mark.skipif(shutil.which(NVCC) is None, reason="no nvcc")
def test_refused_allocations(tmp_path):
    exe = str(tmp_path / "partition_memory")
    subprocess.run([NVCC, "-O1", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "metal4foam_b200", "csrc"), "-o", exe,
                    os.path.join(HERE, "c_abi", "partition_memory.cu"),
                    os.path.join(HERE, "c_abi", "refused_new.cpp")],
                   check=True, capture_output=True, text=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, (res.returncode, res.stdout, res.stderr)
