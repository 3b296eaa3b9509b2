"""Builds a program of tests/host: device headers of the library compiled as host C++ (cuda_host.hpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def run(name, tmp_path, *args):
    """Compiles tests/host/<name>.cpp with the library's float rules and returns what it prints."""
    from supereight2_gb300 import build
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    try:
        cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    except RuntimeError:
        pytest.skip("no CUDA headers")
    exe = str(tmp_path / name)
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-pthread", "-I", cuda, "-o", exe,
                    os.path.join(HERE, "host", name + ".cpp")], check=True)
    return subprocess.run([exe, *args], check=True, capture_output=True, text=True, timeout=300).stdout
