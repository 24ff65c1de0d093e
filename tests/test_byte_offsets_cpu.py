"""Levels beyond the 32-bit byte offsets of the general warp-row sweep are
kept from it (vfs::fits_byte_offsets, compiled for the host)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_bound(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "offsets_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "vfs_v3p2_gb300", "csrc"),
                    os.path.join(HERE, "native", "offsets_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
