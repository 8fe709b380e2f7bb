"""Launch shapes of the Tier-1 forms (csrc/t1_shape.h) on the host."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_t1_shapes(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "t1_shape_test")
    subprocess.run([gxx, "-O2", "-std=c++17", "-o", exe, os.path.join(ROOT, "tests", "t1_shape_test.cpp")], check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=60)
    assert r.returncode == 0 and "ALL OK" in r.stdout, r.stdout
