"""The device memory pool against fakes of the CUDA calls (no GPU): memory is
freed after the device's work is done, once per object, is held while that wait
is refused, and what the pool does not keep is given back at once."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = "/usr/local/cuda/include"


def test_pool_waits_before_it_frees(tmp_path):
    if not shutil.which("g++") or not os.path.isdir(CUDA_INCLUDE):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path / "pool_fakes")
    subprocess.run(["g++", "-std=c++17", "-w", "-x", "c++", "-I", CUDA_INCLUDE, os.path.join(HERE, "pool_fakes.cpp"),
                    "-o", exe, "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
