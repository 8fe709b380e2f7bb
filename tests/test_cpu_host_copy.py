"""The threaded copy of large pictures (csrc/host_copy.h) on the host: whole copies from several
callers at once, with a bound on their threads together."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_host_copy(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "host_copy_test")
    subprocess.run([gxx, "-O2", "-std=c++17", "-pthread", "-o", exe, os.path.join(ROOT, "tests", "host_copy_test.cpp")],
                   check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert r.returncode == 0 and "ALL OK" in r.stdout, r.stdout
