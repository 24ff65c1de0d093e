"""The FP64 -> FP32 rounding of the Krylov kernels (vfs::narrow, integer pipe)
is compiled for the host from the same header and compared with the
compiler's conversion (round to nearest even): at and beside every binary32
value of a stride, at and beside the midpoints, on random doubles of every
exponent and on the special classes."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_narrow_matches_hardware_conversion(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "narrow_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "vfs_v3p2_gb300", "csrc"),
                    os.path.join(HERE, "native", "narrow_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe, "1021"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
