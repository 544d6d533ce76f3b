"""The GEMM's work iterator with the partial wave cut into pieces of K, replayed on the host."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_k_chunks_cover_every_block_exactly_once(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "k_chunks_test")
    src = os.path.join(ROOT, "tests", "native", "k_chunks_test.cu")
    build = subprocess.run([nvcc, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "slowrun_b200", "csrc"), "-gencode",
                            "arch=compute_100a,code=sm_100a", "-o", exe, src], capture_output=True, text=True, timeout=600)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0 and " 0 failures" in run.stdout, run.stdout[-3000:]
