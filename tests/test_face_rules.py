"""Face rules are built on demand (plan.H), checked in C++ without a GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

LIB = os.path.join(ROOT, "chombo_3.2_b200")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_face_rules_are_built_on_demand(tmp_path):
    exe = str(tmp_path / "face_rules_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "face_rules_check.cpp"), "-L" + LIB, "-l:libcmg.so",
                    "-Wl,-rpath," + LIB], check=True)
    out = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert out.returncode == 0 and out.stdout.endswith("ok\n"), out.stdout
