"""A kernel launch that fails leaves no error behind for a later check."""
import os
import shutil
import subprocess

import pytest

from maxmulsk_b200 import build


def test_failed_launch_leaves_no_pending_error(tmp_path):
    if not shutil.which(build.NVCC):
        pytest.skip("no nvcc")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "launch_check.cu")
    exe = str(tmp_path / "launch_check")
    subprocess.run([build.NVCC, *build.CUFLAGS, src, "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["9", "0", "0", "0"]        # cudaErrorInvalidConfiguration, then success
