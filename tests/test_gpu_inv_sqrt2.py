"""The kernels' packed roots equal IEEE ones for every binary32 input in either half."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_packed_roots_every_pattern(rfmm_mod, tmp_path):
    from rfmm import build as B
    exe = str(tmp_path / "inv_sqrt2_check")
    subprocess.run([B.nvcc(), "-std=c++17", "-O3", *B.ARCH, *B.KERNEL_FLAGS, "-I", B.CSRC,
                    os.path.join(REPO, "tests", "native", "inv_sqrt2_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.split() == ["0", "0", "0", "0"], out.stdout
