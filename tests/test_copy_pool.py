"""The server's split host copies: right bytes for any size and number of
threads, and no exception when memory for a copy's bookkeeping is refused."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_copies_are_right_and_never_throw(tmp_path):
    exe = str(tmp_path / "copy_pool_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-pthread",
                    "-I", os.path.join(REPO, "fmm-rainbow_gb300", "csrc"),
                    os.path.join(REPO, "tests", "native", "copy_pool_check.cpp"), "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
