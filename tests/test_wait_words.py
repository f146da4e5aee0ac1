"""A bounded wait that runs out records it in an error word by an atomic, which
works on global or shared memory: the compiler reports one on a local
variable, and the tensor-core kernels must compile without that report."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_atomic_on_local_memory(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src = os.path.join(ROOT, "lowrankapprox.jl_gb300", "csrc", "tc_sketch.cu")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                        "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"), "-c", src, "-o",
                        str(tmp_path / "tc.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "local memory" not in r.stderr + r.stdout
