"""An error that a CUDA call returned is reported once, by the call that met it."""
import os
import subprocess

import pytest

from sbd_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu  # without a driver every call fails, that for the last error too
def test_thrown_errors_are_cleared(tmp_path):
    exe = str(tmp_path / "cuda_error")
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, os.path.join(ROOT, "tests", "cpp", "cuda_error.cu"),
                    "-o", exe, "-lcudart"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
