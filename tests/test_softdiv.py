"""Reciprocals, quotients and square roots on the integer pipe
(fgc_softdiv.cuh): on the CPU against its division and square root
(softdiv_check.cpp), and on the GPU, whose seeds differ, against CUDA's
functions (softdiv_gpu.cu)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_matches_cpu_division(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "softdiv_check")
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-std=c++17", os.path.join(HERE, "softdiv_check.cpp"), "-o",
                    exe], check=True)
    r = subprocess.run([exe, "4000000"], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr


@pytest.mark.gpu
def test_matches_cuda_functions(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "softdiv_gpu")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-std=c++17",
                    "--expt-relaxed-constexpr", os.path.join(HERE, "softdiv_gpu.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
