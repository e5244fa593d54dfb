"""The tables of the coarse cluster launch (coarse.H), checked against the layouts in C++ without a GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

LIB = os.path.join(ROOT, "chombo_3.2_b200")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_coarse_tables_match_the_layouts(tmp_path):
    exe = str(tmp_path / "coarse_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "coarse_check.cpp"), "-L" + LIB, "-l:libcmg.so",
                    "-Wl,-rpath," + LIB], check=True)
    out = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert out.returncode == 0 and out.stdout.endswith("ok\n"), out.stdout
