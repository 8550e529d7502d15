"""The host-side rules of csrc/rules.hpp (tests/cpp/test_rules.cpp, compiled here
with the host C++ compiler: they need no GPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rules(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "test_rules")
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I",
                        os.path.join(ROOT, "magpy_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "test_rules.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "rules ok" in r.stdout, r.stderr
