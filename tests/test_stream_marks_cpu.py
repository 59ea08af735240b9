"""Marks in a stream's work (runtime/stream_mark.h): which of two marks a buffer keeps, which waits are left out, what happens
when no event can be had.  The header is compiled for the host against a stand-in for the CUDA runtime."""
import os
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_stream_marks(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda_include = Path(nvcc).resolve().parent.parent / "include"
    exe = tmp_path / "stream_marks_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(ROOT / "ryft_b200" / "csrc" / "runtime"), "-I", str(cuda_include),
                    str(ROOT / "tests" / "stream_marks_check.cc"), "-o", str(exe)], check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
