"""A failed CUDA call is reported by the call that failed and by no later one."""

import os
import shutil
import subprocess

import numpy as np
import pytest

import skb_cuda

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "spectral-kernel-benchmarks_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def _run(command, exe):
    subprocess.run(command + ["-std=c++17", "-o", str(exe)], check=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip() == "ok"


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_refused_launch_leaves_no_error(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text("")  # the checker's stand-in takes its place
    _run(["g++", "-I", str(tmp_path), "-I", CSRC, os.path.join(ROOT, "tests", "launch_check.cpp")], tmp_path / "check")


@pytest.mark.gpu
def test_refused_launch_then_a_valid_one(tmp_path):
    _run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC, os.path.join(ROOT, "tests", "launch_check.cu")],
         tmp_path / "check")


@pytest.mark.gpu
def test_refused_allocation_does_not_fail_the_next_call():
    """cudaMalloc of more than any device holds is refused on the host; the plain
    launches of the calls after it must not report it again."""
    w = skb_cuda.Workload(16, 16, 5, 2)
    fft = skb_cuda.FFTProvider(w)
    rng = np.random.default_rng(1)
    spectrum = fft.forward(rng.uniform(-1, 1, w.real_elements))
    want = fft.gather_retained(spectrum)
    with pytest.raises(MemoryError):
        skb_cuda.DeviceArray(1 << 46)
    assert np.array_equal(fft.gather_retained(spectrum), want)
