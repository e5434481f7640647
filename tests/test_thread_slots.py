"""The page-locked norm slots of the plain path's threads are handed on from
thread to thread (thread_slots.h, compiled with the host C++ compiler)."""
import os
import shutil
import subprocess

import pytest


def test_threads_hand_their_slots_on(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = str(tmp_path / "slots")
    subprocess.run([cxx, "-O2", "-std=c++17", "-pthread", "-I",
                    os.path.join(root, "block_ipt_gb300", "csrc"),
                    os.path.join(root, "tests", "cpp", "thread_slots.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
