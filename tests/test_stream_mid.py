"""Pieces of the streaming push (csrc/k_stream_mid.cuh) checked on the CPU: a host harness (tests/stream_mid_check.cu) built with
nvcc compares the weights that the gather of the midpoint fields applies with their FP64 values. Where the mixed
form adds an analytic wave or an external element the weights are FP64 and only their products are rounded to FP32. The time of
a half-cell is compared with the form by roots and quotients for particles that run backwards, where gamma + p_z cancels."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "gem-pic-3d_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc is not installed")
def test_pieces_of_the_streaming_push(tmp_path):
    exe = tmp_path / "stream_mid_check"
    subprocess.run([NVCC, "-std=c++17", "-O2", "-I", CSRC, "-I", os.path.join(HERE, "..", "include"), "--expt-relaxed-constexpr",
                    "-o", str(exe), os.path.join(HERE, "stream_mid_check.cu")], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "weights" in r.stdout
