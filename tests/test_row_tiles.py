"""CPU check of the SM-pair kernels' tile lists (fastpath/row_tiles_check.cpp)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SRC = os.path.join(ROOT, "tests", "fastpath", "row_tiles_check.cpp")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_tiles_cover_each_entry_once(tmp_path):
    exe = str(tmp_path / "row_tiles_check")
    # the header's only CUDA include is for the qualifiers the check defines away
    (tmp_path / "cuda_runtime.h").write_text("")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(tmp_path), "-I",
                    os.path.join(ROOT, "qld_b200", "csrc"), "-o", exe, SRC], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout
