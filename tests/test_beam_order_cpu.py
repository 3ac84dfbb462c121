"""The warp's beam (insertion, choice of the next entry, whole searches) with NaN and
infinite distances: the device functions, compiled for the host with one fiber per lane,
against plain sorted lists."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_beam_agrees_with_sorted_lists(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not shutil.which("g++") or not os.path.isfile(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path / "beam")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-isystem", include,
                    os.path.join(HERE, "host_beam.cpp"), "-o", exe], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout + p.stderr
