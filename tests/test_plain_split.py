"""The 56-bit digit split of the plain path's tensor-core product
(oz_biased_any<7> of block_ipt_gb300/csrc/oz.cuh), compiled with the host C++
compiler from the library's own header: digit ranges and the exact value on 3
million entries of every kind."""
import os
import platform
import shutil
import subprocess

import pytest


def test_split_digits(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    if platform.machine() not in ("x86_64", "aarch64"):
        pytest.skip("needs a long double of at least 64 significant bits")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = str(tmp_path / "oz56")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(root, "block_ipt_gb300", "csrc"),
                    os.path.join(root, "tests", "cpp", "oz_digits56.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert "mismatches 0" in out.stdout
