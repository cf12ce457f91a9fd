"""The pool of pinned size records that the waiting calls (iso_*_sync) lease from:
no allocation per thread, none freed at a thread's end, none shared by two calls,
none of a context that has ended.  Plain C++ with fake memory, no GPU."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_size_pool(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "size_pool")
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-pthread", "-I",
                           os.path.join(os.path.dirname(HERE), "isoext_gb300", "csrc"), "-o", exe,
                           os.path.join(HERE, "size_pool.cpp")])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
